"""The kernel that a product without a requested one runs on, as the number of
stored blocks (known, unknown, wrong) and the sizes choose it
(spmm_bcsr_mm_nnzb): each choice gives the product, and its launch can be
captured and replayed, also by two streams at once.

Bound: products of two 16-bit floats are exact in fp32, so a sum of n terms is
off by at most n steps of 2^-23 of the sum of |a| |b|."""
import ctypes

import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def problem(dev, M, K, N, bR, density, dtype, seed):
    rng = np.random.default_rng(seed)
    keep = rng.uniform(size=(M // bR, K // 16)) < density
    keep[1:2] = False
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    g = torch.Generator(device=dev).manual_seed(seed)
    kind = torch.bfloat16 if dtype == m.DType.BF16 else torch.float16
    uniform = lambda *s: (torch.rand(s, generator=g, device=dev) * 2 - 1).to(kind)
    n = int(keep.sum())
    vals, B = uniform(n, bR, 16), uniform(K, N)
    A = m.BCSR(M, K, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]), vals.view(-1),
               dtype)
    Ad = torch.zeros(M // bR, K // 16, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = vals.double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(M, K)
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    bound = terms * 2.0 ** -23 * (Ad.abs() @ B.double().abs())
    return A, B, Ad @ B.double(), bound


# 16 and 32 rows: mma.sync, then long rows; 64 rows: short rows, ordinary ones, 512-column tiles
SHAPES = [(512, 256, 264, 16, 0.3), (512, 512, 264, 16, 0.9), (1024, 512, 136, 32, 0.6), (704, 208, 520, 32, 0.2),
          (1024, 512, 264, 64, 0.15), (1024, 512, 264, 64, 0.8), (64, 64, 40, 64, 0.9), (8192, 64, 1040, 64, 0.7)]


# mma.sync's ring of eight (256-, 128-column tiles, few columns), and tcgen05 for many items
SHAPES += [(512, 512, 264, 16, 0.3), (512, 512, 136, 16, 0.25), (496, 512, 40, 16, 0.4), (512, 1040, 72, 32, 0.5),
           (7424, 256, 512, 32, 0.5), (8192, 256, 512, 16, 0.8)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [m.DType.F16, m.DType.BF16])
@pytest.mark.parametrize("hint", ["right", "unknown", "none", "many"])
def test_default_kernel(dev, shape, dtype, hint):
    M, K, N, bR, density = shape
    A, B, ref, bound = problem(dev, M, K, N, bR, density, dtype, seed=M + N)
    n = {"right": A.nnzb, "unknown": -1, "none": 0, "many": 1 << 40}[hint]
    C = torch.full((M, N), float("nan"), device=dev)
    a = A.desc()
    b = m._lib.DenseDesc(B.data_ptr(), None, 1.0, N)
    m.check(m.lib().spmm_bcsr_mm_nnzb(ctypes.byref(a), n, ctypes.byref(b), N, C.data_ptr(), N, None, m.stream_handle()))
    m.device_error_check()
    assert ((C.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("shape", [SHAPES[1], SHAPES[5], SHAPES[7]])
def test_captured_and_replayed_by_two_streams(dev, shape):
    M, K, N, bR, density = shape
    A, B, ref, bound = problem(dev, M, K, N, bR, density, m.DType.F16, seed=7)
    streams, graphs, Cs = [torch.cuda.Stream(), torch.cuda.Stream()], [], []
    for s in streams:
        C = torch.full((M, N), float("nan"), device=dev)
        m.spmm(A, B, C=C)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            m.spmm(A, B, C=C)
        C.fill_(float("nan"))
        graphs.append(g)
        Cs.append(C)
    torch.cuda.synchronize()
    for _ in range(3):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    m.device_error_check()
    for C in Cs:
        assert ((C.double() - ref).abs() <= bound).all()


# both sides of the lines for 64-row blocks: few blocks, as many items as SMs, whole
# boxes, long rows in many items; split fp16 likewise
LINES = [(576, 640, 104, 64, 0.2), (9664, 256, 128, 64, 0.5), (9664, 256, 136, 64, 0.1), (9792, 128, 64, 64, 0.6),
         (19584, 128, 256, 64, 0.9), (19584, 512, 256, 64, 0.4), (19584, 256, 264, 64, 0.1)]


@pytest.mark.parametrize("shape", LINES)
@pytest.mark.parametrize("dtype", [m.DType.F16, m.DType.F16_SPLIT])
@pytest.mark.parametrize("hint", ["right", "unknown"])
def test_default_kernel_of_64_rows(dev, shape, dtype, hint):
    M, K, N, bR, density = shape
    A, B, ref, bound = problem(dev, M, K, N, bR, density, m.DType.F16, seed=M + N)
    lo = None
    if dtype == m.DType.F16_SPLIT:   # (low halves of zero: the product is the fp16 one)
        A.dtype, A.vals_lo, lo = dtype, torch.zeros_like(A.vals), torch.zeros_like(B)
    C = torch.full((M, N), float("nan"), device=dev)
    a = A.desc()
    b = m._lib.DenseDesc(B.data_ptr(), None if lo is None else lo.data_ptr(), 1.0, N)
    n = A.nnzb if hint == "right" else -1
    m.check(m.lib().spmm_bcsr_mm_nnzb(ctypes.byref(a), n, ctypes.byref(b), N, C.data_ptr(), N, None, m.stream_handle()))
    m.device_error_check()
    assert ((C.double() - ref).abs() <= bound).all()
