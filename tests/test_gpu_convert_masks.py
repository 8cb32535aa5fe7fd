"""Dense -> BCSR with and without the mask workspace, at the edges of a warp's
group of blocks (32 lanes), of a row's groups and of the pieces a block is
copied in: both equal the oracle bit for bit."""
import ctypes

import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,bR,bC", [(16, 16, 16, 16), (16, 16400, 16, 16), (1024, 528, 16, 16), (192, 272, 64, 16),
                                       (96, 1040, 48, 80), (64, 1536, 32, 256)])
@pytest.mark.parametrize("sparsity", [0.999, 0.9, 0.0])
def test_masked_and_rescan_match_oracle(dev, M, K, bR, bC, sparsity):
    A = oracle.f32_to_f16(oracle.generate_matrix(M, K, sparsity, "random", 16, 5))
    exp = oracle.bcsr(A, bR, bC)
    t = torch.from_numpy(A.view(np.float16).copy()).to(dev)
    p, s = (lambda x: ctypes.c_void_p(x.data_ptr())), m.stream_handle()
    L = m.lib()
    for masked in (True, False):
        rp = torch.full((M // bR + 1,), -1, dtype=torch.int32, device=dev)
        masks = torch.empty(L.spmm_dense_to_bcsr_mask_words(M, K, bR, bC), dtype=torch.int32, device=dev)
        n = ctypes.c_longlong(-1)
        if masked:
            m.check(L.spmm_dense_to_bcsr_count_masks(p(t), M, K, K, bR, bC, p(rp), p(masks), ctypes.byref(n), s))
        else:
            m.check(L.spmm_dense_to_bcsr_count(p(t), M, K, K, bR, bC, p(rp), ctypes.byref(n), s))
        ci = torch.full((n.value,), -1, dtype=torch.int32, device=dev)
        v = torch.full((n.value * bR * bC,), float("nan"), dtype=torch.float16, device=dev)
        if n.value and masked:
            m.check(L.spmm_dense_to_bcsr_fill_masks(p(t), M, K, K, bR, bC, p(rp), p(masks), p(ci), p(v), s))
        elif n.value:
            m.check(L.spmm_dense_to_bcsr_fill(p(t), M, K, K, bR, bC, p(rp), p(ci), p(v), s))
        got = rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy().view(np.uint16)
        for g, e in zip(got, exp):
            assert np.array_equal(g, e)
