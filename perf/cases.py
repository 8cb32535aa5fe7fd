"""The work a user has this library do, as cases that can be timed.

A case is a dict of plain values. `kind` names the entry point:

  dropin   the reference-shaped launchers sparseMatrixMulTensor{,32x16,64x16}
  spmm     spmm(A, B) with the library's own choice of kernel
  plan     BcsrPlan: the per-matrix plan of a caller whose matrix stays
  batch    BatchPlan: many uneven products in one launch
  hybrid   the BCSR + CSR product, planned (HcsrPlan) or in one call (hcsr_mm)
  convert  dense_to_bcsr: a dense fp16 matrix into BCSR
  train    one forward and backward pass of the cost model (MLP.loss_grad)

Structures, values and sizes follow the repository's workloads: block heights
16, 32 and 64; random, band, block-diagonal and log-normal structures; values
uniform in [-1, 1], or normal with a magnitude of 10^u per block; M and K of
512 to 16384 and N of 64 to 4096, block densities of 0.5 to 25 %.
"""
import math
import random

import numpy as np
import torch

import matrixmultiplicationcuda_gb300 as m
from matrixmultiplicationcuda_gb300 import costmodel

PATTERNS = ("random", "band", "blockdiag", "lognormal")
DTYPES = {"f16": m.DType.F16, "bf16": m.DType.BF16, "e4m3": m.DType.E4M3, "split": m.DType.F16_SPLIT}
LARGEST_FLOPS = 2.0 * 8192 * 8192 * 0.20 * 4096   # the largest listed product
MLP_IN, MLP_HIDDEN, MLP_LAYERS, MLP_OUT = 18, 64, 3, 56


def listed():
    return [
        # the reference harness's own case: a small product, called one by one
        dict(name="dropin_1024_16x16", kind="dropin", M=1024, K=1024, N=1024, bR=16, pattern="random",
             density=0.10, dtype="f16", values="uniform"),
        # the reference's main kernel at the size of its larger benches
        dict(name="dropin_8192_16x16", kind="dropin", M=8192, K=8192, N=1024, bR=16, pattern="random",
             density=0.05, dtype="f16", values="uniform"),
        # a pruned layer with rows of very different lengths and an N that is no multiple of a tile
        dict(name="spmm_6176_32x16_ragged", kind="spmm", M=6176, K=8176, N=1000, bR=32, pattern="lognormal",
             density=0.05, dtype="f16", values="uniform"),
        # the largest product of the sweep: many columns, dense enough to load the tensor cores
        dict(name="spmm_8192_64x16_wide", kind="spmm", M=8192, K=8192, N=4096, bR=64, pattern="random",
             density=0.20, dtype="bf16", values="uniform"),
        # a fixed large matrix multiplied again and again, inputs in place before the loop: the headline
        dict(name="plan_16384_64x16", kind="plan", M=16384, K=16384, N=512, bR=64, pattern="random",
             density=0.02, dtype="f16", values="scaled", n_tile=512, inputs_ready=True),
        # a banded operator with small blocks on the default plan, B written just before each product
        dict(name="plan_8192_16x16_band", kind="plan", M=8192, K=8192, N=1024, bR=16, pattern="band",
             density=0.05, dtype="bf16", values="uniform", n_tile=0, inputs_ready=False),
        # 8-bit weights and activations with a scale per block
        dict(name="spmm_16384_64x16_e4m3", kind="spmm", M=16384, K=16384, N=512, bR=64, pattern="random",
             density=0.02, dtype="e4m3", values="scaled"),
        # near-fp32 accuracy: B arrives in fp32, is split into two halves and multiplied
        dict(name="spmm_16384_64x16_split", kind="spmm", M=16384, K=16384, N=512, bR=64, pattern="random",
             density=0.02, dtype="split", values="scaled"),
        # the layers of a whole model at once, every one of another size and structure
        dict(name="batch_64_uneven", kind="batch", count=64, specs=2024),
        # dense blocks plus scattered entries, kept as a hybrid matrix
        dict(name="hybrid_4096", kind="hybrid", M=4096, K=4096, N=1024, density=0.10, scatter=0.02, planned=True),
        # a pruned dense weight turned into blocks
        dict(name="convert_8192_16x16", kind="convert", M=8192, K=8192, bR=16, density=0.05),
        # a mini-batch of the cost model's training
        dict(name="train_256", kind="train", batch=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(rng, lo, hi, q):
    return int(min(hi // q, max(-(-lo // q), round(_log(rng, lo, hi) / q)))) * q


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "spmm", "spmm", "spmm", "plan", "plan", "batch", "hybrid", "convert",
                       "train"])
    if kind == "train":
        return dict(kind=kind, batch=int(_log(rng, 16, 2000)))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 64), specs=rng.randint(1, 1 << 20))
    if kind == "convert":
        bR = rng.choice([16, 32, 64])
        return dict(kind=kind, M=_multiple(rng, 512, 8192, bR), K=_multiple(rng, 512, 8192, 16), bR=bR,
                    density=_log(rng, 0.005, 0.25))
    if kind == "hybrid":
        return dict(kind=kind, M=_multiple(rng, 1024, 4096, 16), K=_multiple(rng, 1024, 4096, 16),
                    N=_multiple(rng, 64, 1024, 8), density=_log(rng, 0.02, 0.10), scatter=_log(rng, 0.001, 0.02),
                    planned=rng.random() < 0.5)
    bR = rng.choice([16, 32, 64])
    case = dict(kind=kind, M=_multiple(rng, 512, 16384, bR), K=_multiple(rng, 512, 16384, 16), bR=bR,
                pattern=rng.choice(PATTERNS), density=_log(rng, 0.005, 0.25))
    if kind == "dropin":
        case["dtype"] = "f16"
    elif kind == "plan":
        case["dtype"] = rng.choice(["f16", "bf16"])
        case["n_tile"] = rng.choice([0, 512])
        case["inputs_ready"] = rng.random() < 0.5
    else:
        case["dtype"] = rng.choice(["f16", "f16", "bf16", "e4m3", "split"])
    case["values"] = rng.choice(["uniform", "scaled"])
    # half of the Ns are whole tiles, half are odd ones
    q = rng.choice([64, 16 if case["dtype"] == "e4m3" else 8])
    most = LARGEST_FLOPS / (2.0 * case["M"] * case["K"] * case["density"])
    if case["dtype"] == "split":
        most /= 3
    case["N"] = _multiple(rng, 64, int(max(64, min(4096, most))), q)
    return case


# ---- inputs -------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda") * 2 - 1


def _mask(g, M, K, bR, pattern, density):
    """Which of the (M / bR) x (K / 16) blocks are stored."""
    MB, KB = M // bR, K // 16
    if pattern == "random":
        keep = torch.rand(MB, KB, generator=g, device="cuda") < density
    elif pattern == "lognormal":
        # row counts with mean density * KB and a coefficient of variation of 1.5
        sigma = math.sqrt(math.log(1 + 1.5 ** 2))
        z = torch.randn(MB, generator=g, device="cuda")
        count = (density * KB * torch.exp(sigma * z - sigma * sigma / 2)).round().long().clamp_(0, KB)
        rank = torch.rand(MB, KB, generator=g, device="cuda").argsort(1).argsort(1)
        keep = rank < count[:, None]
    else:
        row = (torch.arange(MB, device="cuda").double() + 0.5)[:, None] * bR
        col = (torch.arange(KB, device="cuda").double() + 0.5)[None, :] * 16
        if pattern == "band":
            keep = (col - row * (K / M)).abs() < max(16.0, density * K / 2)
        else:
            tile = max(64, round(density * K / 64) * 64)
            keep = torch.floor(row / tile) == torch.floor(col / tile)
    keep[0, 0] = True
    return keep


def _structure(keep):
    rp = torch.zeros(keep.shape[0] + 1, dtype=torch.int32, device="cuda")
    rp[1:] = keep.sum(1).cumsum(0)
    return rp, keep.nonzero()[:, 1].to(torch.int32).contiguous()


def _block_values(g, nnzb, bR, values):
    if values == "uniform":
        return _uniform(g, nnzb, bR * 16)
    return torch.randn(nnzb, bR * 16, generator=g, device="cuda") * 10.0 ** (3 * _uniform(g, nnzb, 1))


def _product(case, g):
    """(keep, fp32 block values, fp32 B) of a single product."""
    keep = _mask(g, case["M"], case["K"], case["bR"], case["pattern"], case["density"])
    v = _block_values(g, int(keep.sum()), case["bR"], case["values"])
    B = _uniform(g, case["K"], case["N"]) if case["values"] == "uniform" else \
        torch.randn(case["K"], case["N"], generator=g, device="cuda")
    return keep, v, B


def _batch_specs(case):
    rng = random.Random(case["specs"])
    out = []
    for _ in range(case["count"]):
        size = int(round(rng.uniform(512, 8192) / 64)) * 64
        out.append(dict(M=size, K=size, N=rng.choice([128, 256, 512]), bR=rng.choice([16, 32, 64]),
                        pattern=rng.choice(["random", "band", "blockdiag"]), density=_log(rng, 0.005, 0.25),
                        values="uniform"))
    return out


def _hybrid(case, g):
    """(keep, fp16 block values, element mask of the scattered part, fp16 dense of its values, fp16 B)."""
    keep = _mask(g, case["M"], case["K"], 16, "random", case["density"])
    v = _block_values(g, int(keep.sum()), 16, "uniform").half()
    rest = torch.rand(case["M"], case["K"], generator=g, device="cuda") < case["scatter"]
    rest &= ~keep.repeat_interleave(16, 0).repeat_interleave(16, 1)
    w = _uniform(g, case["M"], case["K"]).half()
    return keep, v, rest, w, _uniform(g, case["K"], case["N"]).half()


def _dense(case, g):
    # as many blocks for every seed: the outputs' sizes depend on it
    MB, KB = case["M"] // case["bR"], case["K"] // 16
    keep = torch.zeros(MB * KB, dtype=torch.bool, device="cuda")
    keep[torch.rand(MB * KB, generator=g, device="cuda").argsort()[:max(1, round(case["density"] * MB * KB))]] = True
    keep = keep.view(MB, KB)
    A = _uniform(g, case["M"], case["K"]).half()
    return keep, A * keep.repeat_interleave(case["bR"], 0).repeat_interleave(16, 1)


def _training(case, seed):
    """Host arrays: parameters (mu, sigma, then each layer's W and b), X, T, mask."""
    rng = np.random.default_rng(int(seed) * 7919 + 17)
    mu, sigma = rng.normal(size=MLP_IN), rng.uniform(0.5, 2.0, MLP_IN)
    dims = [MLP_IN] + [MLP_HIDDEN] * MLP_LAYERS + [MLP_OUT]
    params = [mu, sigma]
    for fan_in, fan_out in zip(dims, dims[1:]):
        params += [(rng.normal(size=(fan_out, fan_in)) * math.sqrt(2.0 / fan_in)).ravel(),
                   rng.normal(size=fan_out) * 0.1]
    n = case["batch"]
    X = mu + sigma * rng.normal(size=(n, MLP_IN))
    T = 3.0 + rng.normal(size=(n, MLP_OUT))
    mask = rng.random((n, MLP_OUT)) < 0.8
    f = np.float32
    return np.concatenate(params).astype(f), X.astype(f), T.astype(f), mask.astype(f)


def _matrix(case, keep, v32, dtype):
    rp, ci = _structure(keep)
    vals, lo, scales = m.quantize(v32.reshape(-1), dtype, block_elems=case["bR"] * 16)
    return m.BCSR(case["M"], case["K"], case["bR"], 16, rp, ci, vals, dtype, lo, scales)


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "train":
        params, X, T, mask = _training(case, seed)
        net = costmodel.MLP(costmodel.shape(n_out=MLP_OUT, n_in=MLP_IN, hidden=MLP_HIDDEN, layers=MLP_LAYERS), params)
        return dict(kind=kind, net=net, X=torch.from_numpy(X).cuda(), T=torch.from_numpy(T).cuda(),
                    mask=torch.from_numpy(mask).cuda())
    if kind == "convert":
        return dict(kind=kind, A=_dense(case, g)[1], bR=case["bR"])
    if kind == "hybrid":
        keep, v, rest, w, B = _hybrid(case, g)
        A = m.BCSR(case["M"], case["K"], 16, 16, *_structure(keep), v.reshape(-1))
        csr = (*_structure(rest), w[rest].contiguous())
        C = torch.empty(case["M"], case["N"], dtype=torch.float32, device="cuda")
        plan = m.HcsrPlan(A, *csr) if case["planned"] else None
        return dict(kind=kind, A=A, csr=csr, plan=plan, B=B, C=C)
    if kind == "batch":
        problems = []
        for spec in _batch_specs(case):
            keep, v, B = _product(spec, g)
            C = torch.empty(spec["M"], spec["N"], dtype=torch.float32, device="cuda")
            problems.append((_matrix(spec, keep, v, m.DType.F16), B.half(), C))
        return dict(kind=kind, plan=m.BatchPlan(problems), C=[p[2] for p in problems])
    keep, v, B32 = _product(case, g)
    dtype = DTYPES[case["dtype"]]
    A = _matrix(case, keep, v, dtype)
    state = dict(kind=kind, A=A, M=case["M"], K=case["K"], N=case["N"], bR=case["bR"], split=case["dtype"] == "split")
    if state["split"]:
        state["B32"] = B32
        return state
    B, _, scale = m.quantize(B32.reshape(-1), dtype)
    state["B"] = B.view(case["K"], case["N"])
    state["b_scale"] = float(scale[0]) if scale is not None else 1.0
    if kind != "spmm":
        state["C"] = torch.empty(case["M"], case["N"], dtype=torch.float32, device="cuda")
    if kind == "plan":
        cfg = m.Config(kernel=2, n_tile=512, acc_buffers=1) if case["n_tile"] == 512 else None
        state["plan"] = m.BcsrPlan(A, case["N"], cfg)
        state["inputs_ready"] = case["inputs_ready"]
    return state


# ---- one pass -------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "dropin":
        launch = {16: m.sparseMatrixMulTensor, 32: m.sparseMatrixMulTensor32x16,
                  64: m.sparseMatrixMulTensor64x16}[s["bR"]]
        A = s["A"]
        return launch(A.row_ptr, A.col_idx, A.vals, s["B"], s["C"], s["M"], s["N"], s["K"])
    if kind == "spmm":
        if s["split"]:
            hi, lo, _ = m.quantize(s["B32"].view(-1), m.DType.F16_SPLIT)
            shape = (s["K"], s["N"])
            return m.spmm(s["A"], hi.view(shape), B_lo=lo.view(shape))
        return m.spmm(s["A"], s["B"], b_scale=s["b_scale"])
    if kind == "plan":
        return s["plan"].run(s["A"], s["B"], C=s["C"], inputs_ready=s["inputs_ready"])
    if kind == "batch":
        s["plan"].run()
        return s["C"]
    if kind == "hybrid":
        if s["plan"] is not None:
            return s["plan"].run(s["B"], C=s["C"])
        return m.hcsr_mm(s["A"], *s["csr"], s["B"], C=s["C"])
    if kind == "convert":
        return m.dense_to_bcsr(s["A"], s["bR"], 16)
    return s["net"].loss_grad(s["X"], s["T"], s["mask"])


# ---- what a pass cannot do without -----------------------------------------------------

def _product_work(c):
    size = {"f16": 2, "bf16": 2, "e4m3": 1, "split": 4}[c.get("dtype", "f16")]
    b_size = 4 if c.get("dtype") == "split" else size   # a split product reads B in fp32
    MB, KB = c["M"] // c["bR"], c["K"] // 16
    nnzb = c["density"] * MB * KB
    touched = KB if c["pattern"] != "random" else KB * (1 - (1 - c["density"]) ** MB)
    entries = nnzb * c["bR"] * 16
    scales = 4 * nnzb if c.get("dtype") == "e4m3" else 0
    return dict(bytes=entries * size + scales + 4 * nnzb + 4 * (MB + 1) + touched * 16 * c["N"] * b_size
                + 4.0 * c["M"] * c["N"], flops=2.0 * entries * c["N"])


def work(case):
    kind = case["kind"]
    if kind == "train":
        dims = [MLP_IN] + [MLP_HIDDEN] * MLP_LAYERS + [MLP_OUT]
        weights = sum(a * b for a, b in zip(dims, dims[1:]))
        params = 2 * MLP_IN + weights + sum(dims[1:])
        n = case["batch"]
        # forward, weight gradients, and input gradients of all layers but the first
        return dict(bytes=4.0 * (n * (MLP_IN + 2 * MLP_OUT) + 2 * params + 1),
                    flops=2.0 * n * (3 * weights - dims[0] * dims[1]))
    if kind == "convert":
        kept = case["density"] * (case["M"] // case["bR"]) * (case["K"] // 16)
        return dict(bytes=2.0 * case["M"] * case["K"] + kept * (case["bR"] * 32 + 4) + 4 * (case["M"] // case["bR"] + 1),
                    flops=0.0)
    if kind == "hybrid":
        blocks = case["density"] * (case["M"] // 16) * (case["K"] // 16)
        rest = case["scatter"] * (1 - case["density"]) * case["M"] * case["K"]
        return dict(bytes=blocks * 516 + rest * 6 + 4.0 * (case["M"] + 1) + 2.0 * case["K"] * case["N"]
                    + 4.0 * case["M"] * case["N"], flops=2.0 * (blocks * 256 + rest) * case["N"])
    if kind == "batch":
        parts = [_product_work(s) for s in _batch_specs(case)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    return _product_work(case)


# ---- the same results in 64 bits -------------------------------------------------------

def _e4m3(x):
    """Rows of x in e4m3, each with the smallest power of two >= max / 448 as its scale."""
    top = x.abs().amax(1, keepdim=True)
    f, e = torch.frexp(top / 448.0)
    e = torch.where(f == 0.5, e - 1, e)
    scale = torch.where(top > 0, torch.ldexp(torch.ones_like(top), e), torch.ones_like(top))
    return (x / scale).to(torch.float8_e4m3fn).double() * scale.double()


def _stored(x, dtype):
    """The values that a product of this type multiplies (rows share an e4m3 scale)."""
    if dtype == "e4m3":
        return _e4m3(x)
    return x.double() if dtype == "split" else x.to(torch.bfloat16 if dtype == "bf16" else torch.float16).double()


def _expand(keep, blocks, bR):
    """The dense matrix of the stored blocks."""
    MB, KB = keep.shape
    full = torch.zeros(MB, KB, bR * 16, dtype=torch.float64, device="cuda")
    full[keep] = blocks.reshape(-1, bR * 16)
    return full.view(MB, KB, bR, 16).permute(0, 2, 1, 3).reshape(MB * bR, KB * 16)


def _product_exact(case, g, dtype):
    keep, v, B = _product(case, g)
    B = _stored(B.reshape(1, -1), dtype).view(B.shape)
    return _expand(keep, _stored(v, dtype), case["bR"]) @ B


def _train_exact(case, seed):
    params, X, T, mask = (torch.from_numpy(a).cuda().double() for a in _training(case, seed))
    params.requires_grad_()
    x = (X - params[:MLP_IN].detach()) / params[MLP_IN:2 * MLP_IN].detach()
    dims = [MLP_IN] + [MLP_HIDDEN] * MLP_LAYERS + [MLP_OUT]
    at = 2 * MLP_IN
    for layer, (fan_in, fan_out) in enumerate(zip(dims, dims[1:])):
        W = params[at:at + fan_in * fan_out].view(fan_out, fan_in)
        at += fan_in * fan_out
        x = x @ W.t() + params[at:at + fan_out]
        at += fan_out
        if layer < MLP_LAYERS:
            x = torch.nn.functional.gelu(x)
    loss = (mask * (x - T) ** 2).sum() / mask.sum()
    loss.backward()
    return loss.detach().reshape(1), params.grad


def exact(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "convert":
        keep, A = _dense(case, g)
        MB, KB = keep.shape
        blocks = A.view(MB, case["bR"], KB, 16).permute(0, 2, 1, 3)[keep]
        return None, None, blocks.reshape(-1).double()
    if kind == "hybrid":
        keep, v, rest, w, B = _hybrid(case, g)
        return (_expand(keep, v.double(), 16) + w.double() * rest) @ B.double()
    if kind == "batch":
        return [_product_exact(spec, g, "f16") for spec in _batch_specs(case)]
    return _product_exact(case, g, case["dtype"])
