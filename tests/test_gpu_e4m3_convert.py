"""The default e4m3 product at sizes where it runs converted to fp16 on the
tcgen05 pipeline (spmm_bcsr_mm_nnzb's rule: at least ten blocks a row, as many
items as CTAs): block scales that fp16 holds and others, part tiles of columns,
rows of odd block counts, empty rows, rows of more than 32 blocks, a leading
dimension above N with NaN bytes beyond it.

The reference forms A as the kernel does, round_fp16(e4m3 * scale), and sums in
FP64. Products of two fp16 are exact in fp32, so a sum of n terms is off by at
most n steps of 2^-23 of the sum of |a| |b|, and B's scale adds one rounding."""
import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bR", [32, 64])
@pytest.mark.parametrize("N,pad,K", [(512, 0, 272), (400, 16, 272), (256, 0, 1040), (768, 0, 256)])
@pytest.mark.parametrize("scales", ["powers", "any"])
def test_converted_product(dev, bR, N, pad, K, scales):
    tiles = -(-N // 256)
    MB, KB = -(-320 // tiles) + 1, K // 16
    rng = np.random.default_rng(N + K + bR)
    keep = rng.uniform(size=(MB, KB)) < 0.9
    keep[3] = False
    keep[5, 1:] = False
    assert keep.sum() >= 10 * MB
    g = torch.Generator(device=dev).manual_seed(N + bR)

    def e4m3(*shape):
        v = torch.randint(0, 256, shape, generator=g, device=dev, dtype=torch.uint8)
        v[(v & 0x7f) == 0x7f] = 0          # no NaN
        return v

    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    n = int(keep.sum())
    vals = e4m3(n, bR, 16)
    if scales == "powers":                  # down to products that are subnormal in fp16
        sc = torch.exp2(torch.randint(-12, 3, (n,), generator=g, device=dev).float())
    else:
        sc = torch.rand(n, generator=g, device=dev) * 0.02 + 1e-4
    A = m.BCSR(MB * bR, K, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]),
               vals.view(-1), m.DType.E4M3, None, sc)
    Bw = torch.full((K, N + pad), 0x7f, dtype=torch.uint8, device=dev)
    Bw[:, :N] = e4m3(K, N)
    C = torch.full((MB * bR, N), float("nan"), device=dev)
    m.spmm(A, Bw[:, :N], N=N, C=C, b_scale=0.75)
    m.device_error_check()
    blocks = (vals.view(torch.float8_e4m3fn).float() * sc[:, None, None]).half().double()
    Ad = torch.zeros(MB, KB, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = blocks
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, K)
    Bd = Bw[:, :N].contiguous().view(torch.float8_e4m3fn).double()
    ref = 0.75 * (Ad @ Bd)
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    bound = 0.75 * terms * 2.0 ** -23 * (Ad.abs() @ Bd.abs()) + 2.0 ** -24 * ref.abs()
    assert ((C.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("N", [144, 256, 400])
def test_sixteen_rows_many_items(dev, N):
    """16-row blocks with at least 2048 items of 256 columns (mma.sync's wider
    tile), empty rows and part tiles; products and bound as above."""
    MB, K, bR = -(-2048 // -(-N // 256)), 160, 16
    rng = np.random.default_rng(N)
    keep = rng.uniform(size=(MB, K // 16)) < 0.4
    keep[::7] = False
    g = torch.Generator(device=dev).manual_seed(N)
    n = int(keep.sum())
    vals = torch.randint(0, 0x7f, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8)
    sc = torch.rand(n, generator=g, device=dev) * 0.02 + 1e-4
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    A = m.BCSR(MB * bR, K, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]),
               vals.view(-1), m.DType.E4M3, None, sc)
    B = torch.randint(0, 0x7f, (K, N), generator=g, device=dev, dtype=torch.uint8)
    C = torch.full((MB * bR, N), float("nan"), device=dev)
    m.spmm(A, B, C=C)
    m.device_error_check()
    Ad = torch.zeros(MB, K // 16, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = (vals.view(torch.float8_e4m3fn).float() * sc[:, None, None]).half().double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, K)
    Bd = B.view(torch.float8_e4m3fn).double()
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    bound = terms * 2.0 ** -23 * (Ad.abs() @ Bd.abs())
    assert ((C.double() - Ad @ Bd).abs() <= bound).all()


@pytest.mark.parametrize("bR", [32, 64])
@pytest.mark.parametrize("N,shape", [(512, "tail"), (1280, "holes"), (256, "runs"), (4096, "ones")])
def test_converted_product_with_many_empty_rows(dev, bR, N, shape):
    """More items without blocks in a row than the item ring has entries: after
    long rows, at the end of the grid, between rows of one block; bound as above."""
    tiles = -(-N // 256)
    MB, KB = max(48, -(-1400 // tiles)), 96
    rng = np.random.default_rng(N + bR)
    keep = rng.uniform(size=(MB, KB)) < 0.7
    if shape == "tail":
        keep[MB // 3:] = False
    elif shape == "holes":
        keep[rng.uniform(size=MB) < 0.5] = False
    elif shape == "runs":                   # five empty rows at the start, then eight at a time
        keep[np.arange(MB) % 16 > 6] = False
        keep[np.arange(MB) % 16 == 15] = True
        keep[1:6] = False
    else:                                   # rows of one block among empty ones
        keep[rng.uniform(size=MB) < 0.4] = False
        keep[rng.uniform(size=MB) < 0.3, 1:] = False
    assert keep.sum() >= 10 * MB and MB * tiles >= 304
    g = torch.Generator(device=dev).manual_seed(N)
    n = int(keep.sum())
    vals = torch.randint(0, 0x7f, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8)
    sc = torch.exp2(torch.randint(-9, 1, (n,), generator=g, device=dev).float())
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    A = m.BCSR(MB * bR, KB * 16, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]),
               vals.view(-1), m.DType.E4M3, None, sc)
    B = torch.randint(0, 0x7f, (KB * 16, N), generator=g, device=dev, dtype=torch.uint8)
    Ad = torch.zeros(MB, KB, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = (vals.view(torch.float8_e4m3fn).float() * sc[:, None, None]).half().double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, KB * 16)
    Bd = B.view(torch.float8_e4m3fn).double()
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    ref, bound = Ad @ Bd, terms * 2.0 ** -23 * (Ad.abs() @ Bd.abs())
    for _ in range(3):
        C = torch.full((MB * bR, N), float("nan"), device=dev)
        m.spmm(A, B, C=C)
        m.device_error_check()
        assert ((C.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("bR,items,K,N,pad", [(32, 460, 400, 400, 16), (64, 460, 208, 768, 0), (32, 384, 640, 512, 0),
                                              (64, 384, 640, 400, 32), (32, 384, 880, 784, 0), (64, 384, 880, 656, 0)])
def test_converted_product_at_the_rule(dev, bR, items, K, N, pad):
    """Sizes just inside spmm_bcsr_mm_nnzb's rule for the conversion (rows of at
    least 10, 16, 24 and 40 blocks), part tiles of columns; bound as above."""
    MB, KB = -(-items // -(-N // 256)), K // 16
    rng = np.random.default_rng(N + K)
    keep = rng.uniform(size=(MB, KB)) < 0.9
    keep[2] = False
    g = torch.Generator(device=dev).manual_seed(N + bR)
    n = int(keep.sum())
    vals = torch.randint(0, 0x7f, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8)
    vals ^= torch.randint(0, 2, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8) << 7
    sc = torch.rand(n, generator=g, device=dev) * 0.02 + 1e-4
    sc[::3] = torch.exp2(torch.randint(-12, 3, (len(sc[::3]),), generator=g, device=dev).float())   # subnormal in fp16
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    A = m.BCSR(MB * bR, K, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]),
               vals.view(-1), m.DType.E4M3, None, sc)
    Bw = torch.full((K, N + pad), 0x7f, dtype=torch.uint8, device=dev)
    Bw[:, :N] = torch.randint(0, 0x7f, (K, N), generator=g, device=dev, dtype=torch.uint8)
    C = torch.full((MB * bR, N), float("nan"), device=dev)
    m.spmm(A, Bw[:, :N], N=N, C=C, b_scale=0.75)
    m.device_error_check()
    Ad = torch.zeros(MB, KB, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = (vals.view(torch.float8_e4m3fn).float() * sc[:, None, None]).half().double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, K)
    Bd = Bw[:, :N].contiguous().view(torch.float8_e4m3fn).double()
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    ref = 0.75 * (Ad @ Bd)
    bound = 0.75 * terms * 2.0 ** -23 * (Ad.abs() @ Bd.abs()) + 2.0 ** -24 * ref.abs()
    assert ((C.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("bR,N", [(16, 144), (16, 4096), (32, 128), (64, 272)])
@pytest.mark.parametrize("per_row", [0, 1, 2, 5])
def test_short_rows(dev, bR, N, per_row):
    """Rows of at most five blocks, which mma.sync takes one by one; bound as above."""
    MB, KB = 160, 12
    rng = np.random.default_rng(N + per_row)
    keep = np.zeros((MB, KB), bool)
    for r in range(MB):
        keep[r, rng.choice(KB, min(KB, max(0, per_row + int(r == 9) * 7 - int(r == 4))), replace=False)] = True
    g = torch.Generator(device=dev).manual_seed(N + bR)
    n = int(keep.sum())
    vals = torch.randint(0, 0x7f, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8)
    sc = torch.rand(n, generator=g, device=dev) * 0.02 + 1e-4
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    A = m.BCSR(MB * bR, KB * 16, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]),
               vals.view(-1), m.DType.E4M3, None, sc)
    B = torch.randint(0, 0x7f, (KB * 16, N), generator=g, device=dev, dtype=torch.uint8)
    C = torch.full((MB * bR, N), float("nan"), device=dev)
    m.spmm(A, B, C=C)
    m.device_error_check()
    Ad = torch.zeros(MB, KB, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = (vals.view(torch.float8_e4m3fn).float() * sc[:, None, None]).half().double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, KB * 16)
    Bd = B.view(torch.float8_e4m3fn).double()
    terms = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None]
    bound = terms * 2.0 ** -23 * (Ad.abs() @ Bd.abs())
    assert ((C.double() - Ad @ Bd).abs() <= bound).all()


@pytest.mark.parametrize("MB,N", [(24, 128), (230, 512)])     # mma.sync, converted
def test_scales_at_the_ends_of_fp16(dev, MB, N):
    """Block scales that take the largest e4m3 value to fp16's largest (146.2 x 448),
    and ones whose products are subnormal there. Against scaled values in FP64: each
    is off by half a step of fp16, 2^-11 of it or 2^-25, and the sums as above."""
    bR, KB = 64, 24
    g = torch.Generator(device=dev).manual_seed(N)
    n = MB * KB
    vals = torch.randint(0, 0x7f, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8)
    vals ^= torch.randint(0, 2, (n, bR, 16), generator=g, device=dev, dtype=torch.uint8) << 7
    sc = torch.where(torch.rand(n, generator=g, device=dev) < 0.5, 146.2, 2.0 ** -20)
    i = lambda t: t.to(torch.int32).contiguous()
    A = m.BCSR(MB * bR, KB * 16, bR, 16, i(torch.arange(MB + 1, device=dev) * KB), i(torch.arange(KB, device=dev).repeat(MB)),
               vals.view(-1), m.DType.E4M3, None, sc)
    B = torch.randint(0, 0x7f, (KB * 16, N), generator=g, device=dev, dtype=torch.uint8)
    C = m.spmm(A, B)
    m.device_error_check()
    Ad = (vals.view(torch.float8_e4m3fn).double() * sc.double()[:, None, None]).view(MB, KB, bR, 16)
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, KB * 16)
    Bd = B.view(torch.float8_e4m3fn).double()
    off = torch.clamp(Ad.abs() * 2.0 ** -11, min=2.0 ** -25)
    bound = off @ Bd.abs() + 16 * KB * 2.0 ** -23 * ((Ad.abs() + off) @ Bd.abs())
    assert ((C.double() - Ad @ Bd).abs() <= bound).all()
