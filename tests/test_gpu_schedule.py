"""schedule 1 (dynamic) together with a number of CTAs per SM: both are kept, and
the products are those of the default (bound: n terms, each exact in fp32, n steps
of 2^-23 of the sum of |a| |b|)."""
import numpy as np
import pytest

import matrixmultiplicationcuda_gb300 as m

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bR", [16, 32, 64])
def test_dynamic_with_fewer_ctas(dev, bR, capfd, monkeypatch):
    MB, K, N = 640, 512, 264
    rng = np.random.default_rng(bR)
    keep = rng.uniform(size=(MB, K // 16)) < rng.choice([0.05, 0.9], size=(MB, 1))
    g = torch.Generator(device=dev).manual_seed(bR)
    uniform = lambda *s: (torch.rand(s, generator=g, device=dev) * 2 - 1).half()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.int32))).to(dev)
    vals, B = uniform(int(keep.sum()), bR, 16), uniform(K, N)
    A = m.BCSR(MB * bR, K, bR, 16, t(np.concatenate([[0], np.cumsum(keep.sum(1))])), t(np.nonzero(keep)[1]), vals.view(-1))
    Ad = torch.zeros(MB, K // 16, bR, 16, dtype=torch.float64, device=dev)
    Ad[torch.from_numpy(keep).to(dev)] = vals.double()
    Ad = Ad.permute(0, 2, 1, 3).reshape(MB * bR, K)
    bound = t(16 * keep.sum(1)).double().repeat_interleave(bR)[:, None] * 2.0 ** -23 * (Ad.abs() @ B.double().abs())
    monkeypatch.setenv("SPMM_DEBUG", "1")
    # (one, as many as fit, one again: a launch's shared memory does not stay the kernel's limit)
    for ctas in (1, 0, 1, 2):
        C = torch.full((MB * bR, N), float("nan"), device=dev)
        m.spmm(A, B, C=C, cfg=m.Config(kernel=2, n_tile=256, schedule=1, ctas_per_sm=ctas))
        m.device_error_check()
        line = capfd.readouterr().err
        assert "dynamic=1" in line and "per_sm=%d " % (ctas or 2) in line, line
        assert ((C.double() - Ad @ B.double()).abs() <= bound).all()
