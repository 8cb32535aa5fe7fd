"""The cost model's fused forward and backward at the edges of its tiles (8
samples) and CTAs (128): forward, loss and gradient against the FP64 oracle,
with targets that are NaN where the mask is zero. Networks whose weights do
not fit in shared memory run layer by layer and give the same. Bars: fp32 sums
of at most 1024 terms through at most 17 layers stay within 1e-5 of the largest
output, and the gradient's batch sums within 1e-4 of its largest entry."""
import numpy as np
import pytest

from matrixmultiplicationcuda_gb300 import costmodel
from oracle import mlp_oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(18, 64, 3, 56), (3, 5, 2, 6), (4, 4, 1, 1), (128, 128, 2, 70),
                                  (128, 128, 4, 1024)])
@pytest.mark.parametrize("batch", [1, 7, 8, 9, 1024, 1025])
def test_fused_step_matches_oracle(dev, dims, batch):
    n_in, hidden, layers, n_out = dims
    rng = np.random.default_rng(batch)
    s = costmodel.shape(n_out=n_out, n_in=n_in, hidden=hidden, layers=layers)
    p = costmodel.init_params(s, rng.standard_normal(n_in), rng.uniform(0.5, 2.0, n_in), seed=1)
    X = rng.standard_normal((batch, n_in)).astype(np.float32)
    T = rng.standard_normal((batch, n_out)).astype(np.float32)
    M = (rng.uniform(size=T.shape) > 0.25).astype(np.float32)
    odims = mlp_oracle.dims_of(*dims)
    net = costmodel.MLP(s, p, device=dev)
    Y = net.forward(torch.from_numpy(X).to(dev)).cpu().numpy()
    ref = mlp_oracle.forward(odims, p, X)
    assert np.abs(Y - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    seen = T.copy()
    seen[M == 0] = np.nan
    loss, g = net.loss_grad(*(torch.from_numpy(a).to(dev) for a in (X, seen, M)))
    rl, rg = mlp_oracle.loss_grad(odims, p.astype(np.float64), X, T, M)
    g = g.cpu().numpy()
    assert abs(float(loss) - rl) <= 1e-5 * max(1.0, abs(rl))
    assert np.all(g[:2 * n_in] == 0)
    assert np.abs(g - rg).max() <= 1e-4 * max(np.abs(rg).max(), 1e-30)
