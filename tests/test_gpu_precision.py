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


# the kernel's number in a tuning file, its names, a layer: sums of 576, 1600 and 2304 products
@pytest.mark.parametrize("choice,variants,n,c,k,h,ks", [(6, {"columns"}, 6, 64, 32, 40, 3), (7, {"columns pair"}, 6, 64, 64, 40, 3), (6, {"columns"}, 4, 64, 16, 30, 5),
                                                        (5, {"tap pair", "tap pair cut"}, 128, 256, 256, 14, 3), (5, {"tap pair"}, 20, 64, 128, 28, 5)])
def test_columns_and_pairs_against_float64(tmp_path, choice, variants, n, c, k, h, ks):
    """The columns kernel and the per-tap kernel on pairs are no further from float64 than the one-CTA per-tap kernel: the same products, added in
    float32.  What the order of the sums adds is below one rounding per product, 2^-24, times the square root of their number."""
    rs = np.random.RandomState(k + ks)
    x = rs.standard_normal((n, c, h, h)).astype(np.float32)
    w = (rs.standard_normal((k, c, ks, ks)) / np.sqrt(c * ks * ks)).astype(np.float32)
    want = O.conv2d(x[:3].astype(np.float64), w.astype(np.float64), border_mode="half", subsample=(1, 1), real="double")
    assert want.dtype == np.float64
    path, errors, results = str(tmp_path / "t"), {}, {}
    first = shim.Context(0)
    shim.device_conv2d(T.from_host(first, x, "nhwc"), T.from_host(first, w), border_mode="half")
    first.tuning_save(path)
    first.close()
    head, *rest = open(path).read().splitlines()
    for value in (0, choice):
        open(path, "w").write("\n".join([head] + [" ".join(r.split()[:2] + [str(value)]) for r in rest if r.startswith("a 3.")]) + "\n")
        ctx = shim.Context(0)
        assert ctx.tuning_load(path) == 1
        y = shim.device_conv2d(T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), border_mode="half").to_host()
        assert ctx.last_variant in (variants if value else {"tap"})
        results[value], errors[value] = y, rel(y[:3], want)
        ctx.close()
    order = 2.0 ** -24 * np.sqrt(c * ks * ks)
    assert errors[choice] < BOUND and errors[choice] <= errors[0] + order, errors
    assert rel(results[choice], results[0].astype(np.float64)) <= 2 * order
