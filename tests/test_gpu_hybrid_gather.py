"""The planned hybrid product's gather blocks at the edges of their row copies:
column counts around the 256-column tile, a leading dimension above N with NaN
beyond it, block rows whose last gather block is full or nearly empty, and one
matrix without stored blocks.

Bound: fp16 products are exact in fp32, so a sum of n terms is off by at most
n rounding steps of 2^-23 relative to the sum of |a| |b| (one step a term,
twice fp32's half-unit for an accumulator that truncates), each element."""
import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tile", [256, 512])
@pytest.mark.parametrize("N,pad", [(8, 0), (248, 8), (256, 0), (264, 24), (520, 0), (1016, 8)])
@pytest.mark.parametrize("stored", [0.0, 0.15])
def test_gather_edges(dev, N, pad, stored, n_tile):
    M, K = 176, 208
    rng = np.random.default_rng(N + n_tile)
    keep = rng.uniform(size=(M // 16, K // 16)) < stored
    blocks = np.repeat(np.repeat(keep, 16, 0), 16, 1)
    rest = (rng.uniform(size=(M, K)) < 0.05) & ~blocks
    for br, entries in enumerate([0, 1, 15, 16, 17, 32, 33]):   # rest: as they fall
        free = np.flatnonzero(~blocks[16 * br:16 * br + 16].ravel())
        pick = np.zeros(16 * K, bool)
        pick[rng.permutation(free)[:entries]] = True
        rest[16 * br:16 * br + 16] = pick.reshape(16, K)
    A = rng.uniform(-1, 1, (M, K)).astype(np.float16)
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).astype(dt)).to(dev)
    ptr = lambda mask: np.concatenate([[0], np.cumsum(mask.sum(1))])
    vals = A.reshape(M // 16, 16, K // 16, 16).transpose(0, 2, 1, 3)[keep]
    Ab = m.BCSR(M, K, 16, 16, t(ptr(keep), np.int32), t(np.nonzero(keep)[1], np.int32), t(vals.ravel(), np.float16))
    plan = m.HcsrPlan(Ab, t(ptr(rest), np.int32), t(np.nonzero(rest)[1], np.int32), t(A[rest], np.float16))
    Bw = torch.full((K, N + pad), float("nan"), dtype=torch.float16, device=dev)
    Bw[:, :N] = t(rng.uniform(-1, 1, (K, N)), np.float16)
    C = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev)
    plan.run(Bw[:, :N], N=N, C=C, cfg=m.Config(kernel=2, n_tile=n_tile, schedule=1))
    m.device_error_check()
    plan.close()
    Ad = (A * (blocks | rest)).astype(np.float64)
    Bd = Bw[:, :N].cpu().double().numpy()
    terms = 16 * keep.repeat(16, 0).sum(1) + np.add.reduceat(rest.sum(1), np.arange(0, M, 16)).repeat(16)
    bound = terms[:, None] * 2.0 ** -23 * (np.abs(Ad) @ np.abs(Bd))
    assert (np.abs(C.cpu().numpy() - Ad @ Bd) <= bound).all()


@pytest.mark.parametrize("N", [8, 248, 256, 520])
def test_csr_part_in_one_launch_or_two(dev, N):
    """The unplanned product on both sides of the size at which the CSR part
    gets a launch of its own (M N = 2^18), with rows and block rows that have
    no entries, rows of more than 32 entries and a leading dimension above N."""
    M, K = 1040, 336
    rng = np.random.default_rng(N)
    keep = rng.uniform(size=(M // 16, K // 16)) < 0.2
    blocks = np.repeat(np.repeat(keep, 16, 0), 16, 1)
    rest = (rng.uniform(size=(M, K)) < 0.03) & ~blocks
    rest[32:80] = False
    rest[7] = ~blocks[7]
    A = rng.uniform(-1, 1, (M, K)).astype(np.float16)
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).astype(dt)).to(dev)
    ptr = lambda mask: np.concatenate([[0], np.cumsum(mask.sum(1))])
    vals = A.reshape(M // 16, 16, K // 16, 16).transpose(0, 2, 1, 3)[keep]
    Ab = m.BCSR(M, K, 16, 16, t(ptr(keep), np.int32), t(np.nonzero(keep)[1], np.int32), t(vals.ravel(), np.float16))
    B = t(rng.uniform(-1, 1, (K, N)), np.float16)
    Cw = torch.full((M, N + 8), float("nan"), dtype=torch.float32, device=dev)
    m.hcsr_mm(Ab, t(ptr(rest), np.int32), t(np.nonzero(rest)[1], np.int32), t(A[rest], np.float16), B, N=N, C=Cw)
    m.device_error_check()
    assert torch.isnan(Cw[:, N:]).all()
    Ad = (A * (blocks | rest)).astype(np.float64)
    Bd = B.cpu().double().numpy()
    terms = (16 * keep.repeat(16, 0).sum(1) + rest.sum(1) + 1)[:, None]   # (the two parts' sums are added once)
    bound = terms * 2.0 ** -23 * (np.abs(Ad) @ np.abs(Bd))
    assert (np.abs(Cw[:, :N].cpu().numpy() - Ad @ Bd) <= bound).all()
