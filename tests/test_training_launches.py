"""Training's programmatic launches (cleo_b200/csrc/mlp.cu, launch_step): consecutive kernels are on
the GPU together, so what one writes another may not declare unaliased and constant; and a training
call equals the same steps taken one gradient at a time, each waited for on the host."""
import math
import os
import re

import numpy as np
import pytest

from cleo_b200 import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("kernel,shared", [
    ("k_mlp_fwdbwd", ["params", "partial", "loss_partial"]),
    ("k_mlp_adam", ["params", "m", "v", "partial", "loss_partial"])])
def test_no_restrict_on_what_an_overlapping_kernel_writes(kernel, shared):
    with open(os.path.join(ROOT, "cleo_b200", "csrc", "mlp.cu")) as f:
        args = re.search(kernel + r"\(([^)]*)\)\s*\{", f.read()).group(1)
    by_name = {a.split()[-1].lstrip("*"): a for a in args.split(",")}
    for name in shared:
        assert "__restrict__" not in by_name[name], by_name[name]


M64 = (1 << 64) - 1
GOLDEN = 0x9E3779B97F4A7C15


def _mix(z):
    z = np.asarray(z, dtype=np.uint64)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _samples(seed, step, batch, n):
    """The training kernel's draw: sample of each slot of a step's minibatch, from [0, n)."""
    with np.errstate(over="ignore"):
        key = int(_mix(int(_mix((seed + GOLDEN) & M64)) ^ ((step << 32) | 0x4D4C50)))
        u = _mix(np.uint64(key) + (np.arange(batch, dtype=np.uint64) + np.uint64(1))
                 * np.uint64(GOLDEN))
    hi, lo, n = u >> np.uint64(32), u & np.uint64(0xFFFFFFFF), np.uint64(n)
    return ((hi * n + ((lo * n) >> np.uint64(32))) >> np.uint64(32)).astype(np.int64)


def _data(n):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    gen = torch.Generator(device="cuda").manual_seed(n)
    feats = torch.randn(n, abi.MLP_NFEATURES, device="cuda", generator=gen)
    return feats, torch.randn(n, device="cuda", generator=gen)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,n", [(640, 100_003), (8192, 100_003), (64 * 296 + 128, 50_000)])
def test_training_equals_its_steps_one_by_one(batch, n):
    """Below and above the number of resident CTAs. Adam in float32, operation by operation as the
    update kernel has it: the same bits."""
    from cleo_b200.surrogate import Surrogate
    feats, target = _data(n)
    steps, lr, seed = 12, float(np.float32(2e-3)), 77
    run = Surrogate(seed=9, lib=abi.load_library())
    p, norm = run.get_params()
    losses = run.train(feats, target, steps=steps, batch=batch, lr=lr, seed=seed).cpu().numpy()
    one = Surrogate(seed=9, lib=abi.load_library())
    f32 = np.float32
    b1, b2 = f32(0.9), f32(0.999)
    m, v = np.zeros_like(p), np.zeros_like(p)
    warm = steps // 50 + 1
    for s in range(steps):
        one.set_params(p, norm)
        j = _samples(seed, s, batch, n)
        g, loss = one.loss_grad(feats[j].contiguous(), target[j].contiguous())
        g = g.cpu().numpy()
        assert loss.cpu().numpy()[0] == losses[s]
        f = 0.02 + 0.98 * 0.5 * (1.0 + math.cos(3.141592653589793 * s / steps))
        if s < warm:
            f *= (s + 1) / warm
        bc1, bc2 = 1.0 - 0.9 ** (s + 1), 1.0 - 0.999 ** (s + 1)
        rate, eps = f32(lr * f * math.sqrt(bc2) / bc1), f32(1e-8 * math.sqrt(bc2))
        m = b1 * m + (f32(1) - b1) * g
        v = b2 * v + (f32(1) - b2) * g * g
        p = p - rate * m / (np.sqrt(v) + eps)
    assert np.array_equal(run.get_params()[0].view(np.uint32), p.view(np.uint32))
    run.close()
    one.close()


@pytest.mark.gpu
def test_long_training_twice():
    from cleo_b200.surrogate import Surrogate
    feats, target = _data(200_001)
    out = []
    for _ in range(2):
        s = Surrogate(seed=4, lib=abi.load_library())
        losses = s.train(feats, target, steps=2000, batch=8192, seed=5).cpu().numpy()
        out.append((losses, s.get_params()[0]))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
