"""The batched launch's ring at the edges of its groups (four 16- or 32-row
blocks, three 64-row ones) and of the column indices staged at a time (32, or
30 for 64-row blocks): block rows of every such length, mixed in one launch,
twice, against the FP64 product of the stored values. Bar: fp32 sums of at most
1024 terms, 2e-5 of the largest entry (the table sweep's)."""
import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 4, 5, 8, 9, 12, 13, 29, 30, 31, 32, 33, 34, 59, 60, 61, 63, 64, 0]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("N", [72, 128, 320])
def test_row_lengths_at_group_edges(dev, dtype, N):
    K, rng = 1024, np.random.default_rng(N)
    dt, tt = (m.DType.F16, torch.float16) if dtype == "f16" else (m.DType.BF16, torch.bfloat16)
    problems, refs = [], []
    for bR in (16, 32, 64, 64, 16):
        lengths = rng.permutation(LENGTHS)
        rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
        ci = np.concatenate([np.sort(rng.choice(K // 16, n, replace=False)) for n in lengths]).astype(np.int32)
        v = torch.from_numpy(rng.uniform(-1, 1, len(ci) * bR * 16).astype(np.float32)).to(tt)
        B = torch.from_numpy(rng.uniform(-1, 1, (K, N)).astype(np.float32)).to(tt)
        M = bR * len(lengths)
        A = m.BCSR(M, K, bR, 16, torch.from_numpy(rp).to(dev), torch.from_numpy(ci).to(dev), v.to(dev), dt)
        problems.append((A, B.to(dev), torch.full((M, N), float("nan"), device=dev)))
        refs.append(oracle.bcsr_matmul_f64(rp, ci, v.double().numpy(), bR, 16, B.double().numpy()))
    plan = m.BatchPlan(problems)
    for _ in range(2):
        for _, _, C in problems:
            C.fill_(float("nan"))
        plan.run()
        m.device_error_check()
        for (_, _, C), ref in zip(problems, refs):
            mx, fr = oracle.rel_errors(C.cpu().numpy(), ref)
            assert mx <= 2e-5 and fr <= 2e-5
    plan.close()
