"""Errors against float64 where reductions are cut into more slices than before, or several kernels may run: the rounding of
the operands to TF32 explains them, the order of the sums adds next to nothing."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor

# TF32 drops 13 mantissa bits of each factor: at most 2^-10 relative, 2^-11 * E(1/m) = 0.72 * 2^-11 on average for
# mantissas m in [1, 2), and with the same sign for all, so a sum of products is small by about 1.44 * 2^-11 = 7.0e-4
# (measured 7.7e-4).  The sum itself may add up to the next power of two: 2^-10 = 9.8e-4.
BOUND = 2.0 ** -10


def rel(a, b):
    a = a.astype(np.float64)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("tuned", [False, True], ids=["model", "timed"])
@pytest.mark.parametrize("n,c,k,h,g", [(64, 256, 256, 28, 32), (32, 96, 48, 28, 12), (16, 64, 64, 56, 1)], ids=["g32", "g12", "g1"])
def test_grad_weights_against_float64(tuned, n, c, k, h, g):
    rs = np.random.RandomState(g)
    x, dy = (rs.standard_normal((n, m, h, h)).astype(np.float32) for m in (c, k))
    kw = dict(border_mode="half", num_groups=g)
    want = O.conv2d_grad_weights(x.astype(np.float64), dy.astype(np.float64), (3, 3), real="double", **kw)
    assert want.dtype == np.float64
    ctx = shim.Context(0)
    ctx.set_autotune(tuned)
    X, DY = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, dy, "nhwc")
    for _ in range(2):
        assert rel(shim.device_grad_weights(X, DY, (3, 3), **kw).to_host(), want) < BOUND
    ctx.close()


@pytest.mark.parametrize("tuned", [False, True], ids=["model", "timed"])
@pytest.mark.parametrize("n", [1, 8])
def test_a_stack_of_layers_against_float64(tuned, n):
    """Layers of one image (split reductions) and of eight (pairs of CTAs), each on the result of the one before: every
    layer adds at most the error of its own."""
    rs = np.random.RandomState(n)
    x = rs.standard_normal((n, 256, 28, 28)).astype(np.float32)
    ctx = shim.Context(0)
    ctx.set_autotune(tuned)
    X, exact = T.from_host(ctx, x, "nhwc"), x.astype(np.float64)
    for layer, k in enumerate((256, 512, 512, 512), 1):
        w = (rs.standard_normal((k, exact.shape[1], 3, 3)) * np.sqrt(2.0 / (exact.shape[1] * 9))).astype(np.float32)
        b = rs.standard_normal(k).astype(np.float32) * np.float32(0.05)
        W, B = T.from_host(ctx, w), T.from_host(ctx, b.reshape(1, k, 1, 1))
        X = shim.device_conv2d(X, W, bias=B, relu=True, border_mode="half")
        exact = np.maximum(O.conv2d(exact, w.astype(np.float64), border_mode="half", subsample=(1, 1), real="double") + b.astype(np.float64)[None, :, None, None], 0)
        assert exact.dtype == np.float64 and rel(X.to_host(), exact) < layer * BOUND
    ctx.close()
