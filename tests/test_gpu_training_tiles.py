"""The gradient kernel's tiles (cleo_b200/csrc/mlp.cu): sample counts at the edges of a tile of 64,
one tile a CTA and several, against the FP64 restatement.

Bar, per parameter group, in units of the group's largest sum of the samples' absolute
contributions (what rounding scales with): each contribution carries the error of dot products of
up to 64 terms through two layers and back, below 3 x 64 x 2^-24 = 1.2e-5, and the sums over 64
samples a tile, a few tiles and some 300 CTAs in groups of 16 add below 100 x 2^-24 = 6e-6."""
import numpy as np
import pytest

import mlp_numpy as M
from cleo_b200 import abi
from cleo_b200.surrogate import Surrogate

pytestmark = pytest.mark.gpu


def _absolute_sums(p, norm, feats, target):
    """The mean squared error's gradient and the sums of its terms' magnitudes."""
    W1, b1, W2, b2, W3, b3 = M.unpack(p)
    x, t = M.standardise(feats, target, norm)
    a1 = x @ W1.T + b1
    h1 = M.gelu(a1)
    a2 = h1 @ W2.T + b2
    dy = 2.0 * np.abs(M.gelu(a2) @ W3 + b3 - t) / len(t)
    da2 = dy[:, None] * np.abs(W3[None, :] * M.gelu_grad(a2))
    da1 = (da2 @ np.abs(W2)) * np.abs(M.gelu_grad(a1))
    return {"W1": (da1.T @ np.abs(x)).max(), "b1": da1.sum(0).max(),
            "W2": (da2.T @ np.abs(h1)).max(), "b2": da2.sum(0).max(),
            "W3": (np.abs(M.gelu(a2)).T @ dy).max(), "b3": dy.sum()}


@pytest.mark.parametrize("n", [1, 63, 64, 65, 200, 64 * 296, 64 * 296 + 1, 64 * 700 + 63])
def test_gradient_at_tile_edges(n):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    gen = torch.Generator(device="cuda").manual_seed(n)
    feats = torch.randn(n, 7, device="cuda", generator=gen)
    target = torch.randn(n, device="cuda", generator=gen)
    sur = Surrogate(seed=5, lib=abi.load_library())
    p, norm = sur.get_params()
    g, loss = sur.loss_grad(feats, target)
    g2, _ = sur.loss_grad(feats, target)
    assert torch.equal(g, g2)  # a fixed order of additions
    f, t = feats.cpu().numpy(), target.cpu().numpy()
    l64, g64 = M.loss_grad(p, norm, f, t)
    scale = _absolute_sums(p, norm, f, t)
    g = g.cpu().numpy()
    for name, (a, b) in M.GROUPS.items():
        err = np.max(np.abs(g[a:b] - g64[a:b]))
        assert err <= 1.8e-5 * scale[name], (name, err, scale[name])
    assert abs(float(loss) - l64) <= 1.8e-5 * l64
    sur.close()
