"""The tensor-core inference's pairs of units and its quick GELU (cleo_b200/csrc/mlp.cuh) against the
FP32 check path, which takes the hidden layer one unit at a time with erff: activations from nearly
linear to far in both tails, the reach of the quick exponential's argument, and infinities.

Bar: both paths multiply the same BF16 hidden values, so what may differ is layer 2's FP32 sums of 64
products and the bias (at most 66 x 2^-23 of their absolute sum in either path, truncated or
rounded), the GELU (1e-6 |a|, and its slope is below 1.13) and the last sum of 64. One hidden unit
rounded to another BF16 value moves the sum by 2^-8 of its product, as much as the whole bar for a
unit of average size."""
import numpy as np
import pytest

import mlp_numpy as M
from cleo_b200 import abi
from cleo_b200.surrogate import Surrogate

pytestmark = pytest.mark.gpu


def _bf16(x):
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16 << 16).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("scale", [1e-4, 0.1, 1.0, 6.0, 40.0, 1e6])
def test_pairs_of_units_match_single_ones(scale):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    n = 20011
    gen = torch.Generator(device="cuda").manual_seed(3)
    f = scale * torch.randn(n, 7, device="cuda", generator=gen)
    sur = Surrogate(seed=4, lib=abi.load_library())
    p, nrm = sur.get_params()
    nrm[:7], nrm[7:14], nrm[14], nrm[15] = 0.0, 1.0, 0.0, 1.0
    sur.set_params(p, nrm)
    y = [sur.infer(f, path).cpu().numpy().astype(np.float64)
         for path in (abi.MLP_TCGEN05, abi.MLP_FP32)]
    W1, b1, W2, b2, W3, b3 = M.unpack(p)
    h = np.abs(M.gelu(f.cpu().numpy().astype(np.float64) @ _bf16(W1).T.astype(np.float64) + b1))
    s = h @ np.abs(_bf16(W2)).T.astype(np.float64) + np.abs(b2)   # layer 2's absolute sums
    w3 = np.abs(W3)
    bar = (1.13 * 2 * 66 * 2.0 ** -23 * s + 2e-6 * s) @ w3
    bar += 2 * 66 * 2.0 ** -24 * (s @ w3 + np.abs(b3))
    assert np.all(np.isfinite(y[0])) and np.all(np.abs(y[0] - y[1]) <= bar), \
        np.max(np.abs(y[0] - y[1]) / bar)
    f[7, 2], f[8, 3], f[9, 1] = np.inf, -np.inf, np.nan
    for path in (abi.MLP_TCGEN05, abi.MLP_MMA_SYNC, abi.MLP_FP32):
        bad = ~np.isfinite(sur.infer(f, path).cpu().numpy())
        assert np.array_equal(np.nonzero(bad)[0], [7, 8, 9]), path
    sur.close()
