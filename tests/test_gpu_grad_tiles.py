"""Gradient kernel of the planner's MLP at the edges of its tiles.

64-sample tiles over at most 148 CTAs; up to 16,384 samples one CTA zeroes the
gradient and counts the mask, above that memsets and a counting kernel do; the
final adds are 16-byte vectors where the gradient is so aligned. Against the
float64 oracle with the tolerance of tests/test_gpu_planner.py:
|g_dev - g_ref| <= 1e-3 * max|g_ref| + 1e-4 * |g_ref| (FP32 sums of at most a
few hundred terms per thread: a few 1e-5 of the largest, the rest is room for
samples within rounding of a ReLU's kink).
"""
import numpy as np
import pytest

import adabool_b200 as ab
from adabool_b200 import _native as N
from adabool_b200 import planner as P
from oracle import planner_oracle as PO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 148 * 64, 148 * 64 + 1, 16384, 16385])
@pytest.mark.parametrize("shift", [0, 1])
def test_gradient_at_tile_edges(dev, n, shift):
    import torch
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, 16)).astype(np.float32)
    t = rng.normal(3, 1, (n, 3)).astype(np.float32)
    mask = (rng.random((n, 3)) < 0.8).astype(np.float32)
    mask[0, 0] = -2.0  # any non-zero value counts once
    p = P.init_params(np.zeros(16), np.ones(16), seed=n)
    p[PO.OFF["b1"]:PO.OFF["W2"]] = rng.normal(0, 0.1, 64)
    p[PO.OFF["b2"]:PO.OFF["W3"]] = rng.normal(0, 0.1, 64)

    def shifted(a):  # `shift` floats past a 16-byte boundary
        d = torch.full((a.size + 4,), 7.0, dtype=torch.float32, device="cuda")
        d[shift:shift + a.size] = torch.from_numpy(a.ravel())
        return d, d[shift:shift + a.size]

    (_, dp), (_, dx), (_, dt), (_, dm) = (shifted(a) for a in (p, x, t, mask))
    whole, g = shifted(np.ones(N.PLANNER_PARAMS, np.float32))  # stale values are overwritten
    loss = torch.full((2,), 9.0, dtype=torch.float32, device="cuda")
    for _ in range(2):
        N.check(ab.lib().abf_mlp_grad(N.ptr(dp), N.ptr(dx), N.ptr(dt), N.ptr(dm), n, N.ptr(g), N.ptr(loss), None))
    torch.cuda.synchronize()
    g_ref, l_ref = PO.grad(p, x, t, mask)
    gd = g.cpu().numpy().astype(np.float64)
    assert np.all(np.abs(gd - g_ref) <= 1e-3 * np.abs(g_ref).max() + 1e-4 * np.abs(g_ref)), np.abs(gd - g_ref).max()
    assert abs(loss[0].item() - l_ref) <= 1e-4 * max(l_ref, 1.0)
    assert loss[1].item() == float((mask != 0).sum())
    assert not gd[:32].any()
    around = whole.cpu().numpy()
    assert np.all(around[:shift] == 7.0) and np.all(around[shift + g.numel():] == 7.0)
