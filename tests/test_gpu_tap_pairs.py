"""The per-tap kernel on pairs of CTAs: odd numbers of pixel tiles, filters off the tile widths, several views, groups, outputs with
strides, and tiles whose reduction is cut over several pairs."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
T = shim.DeviceTensor
F = np.float32


@pytest.fixture
def ctx():
    c = shim.Context(0)
    c.set_autotune(False)
    yield c
    c.close()


def tol(dtype):
    return 5e-3 if dtype == F else 2e-2            # the repository's bounds for TF32 factors and float16 tensors


# images and size, channels, filters, kernel, stride, dilation, groups
LAYERS = [(61, 14, 40, 128, 3, 1, 1, 1), (25, 19, 64, 192, 3, 1, 1, 1), (9, 33, 33, 256, 1, 1, 1, 1), (60, 28, 48, 128, 3, 2, 1, 1),
          (13, 28, 64, 320, 2, 1, 3, 1), (21, 15, 128, 256, 3, 1, 1, 2), (10, 70, 64, 512, 5, 3, 1, 1), (150, 7, 96, 384, 3, 1, 1, 1)]


@DTYPES
@pytest.mark.parametrize("n,h,c,k,ks,s,d,g", LAYERS)
def test_against_the_oracle(ctx, dtype, n, h, c, k, ks, s, d, g):
    rs = np.random.RandomState(n + k)
    kw = dict(border_mode="half", subsample=(s, s), filter_dilation=(d, d), num_groups=g)
    x = rs.standard_normal((n, c, h, h)).astype(dtype)
    w = (rs.standard_normal((k, c // g, ks, ks)) / np.sqrt(c // g * ks * ks)).astype(dtype)
    b = rs.standard_normal((1, k, 1, 1)).astype(dtype)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    y = shim.device_conv2d(X, W, bias=B, relu=True, flags=shim.NO_SLAB, **kw)
    assert ctx.last_variant.startswith("tap pair")
    ref = np.maximum(O.conv2d(x.astype(F), w.astype(F), **kw) + b.astype(F), 0)
    assert O.rel_err(y.to_host().astype(F), ref) < tol(dtype)
    plain = shim.device_conv2d(X, W, flags=shim.NO_SLAB, **kw).to_host()
    ctx.set_pair_kernels(False)
    one = shim.device_conv2d(X, W, flags=shim.NO_SLAB, **kw).to_host()
    assert "pair" not in ctx.last_variant
    assert O.rel_err(plain.astype(F), one.astype(F)) < (1e-5 if dtype == F else 1e-3)      # the same products, sums in another order


@DTYPES
def test_strided_gradient_by_class(ctx, dtype):
    """The classes of a strided gradInputs are outputs with strides."""
    rs = np.random.RandomState(3)
    kw = dict(border_mode="half", subsample=(2, 2))
    w = (rs.standard_normal((64, 192, 3, 3)) / 24).astype(dtype)
    dy = rs.standard_normal((48, 64, 14, 15)).astype(dtype)
    W, DY = T.from_host(ctx, w), T.from_host(ctx, dy, "nhwc")
    dx = shim.device_grad_inputs(W, DY, (28, 29), flags=shim.NO_SLAB | shim.NO_MERGE_PARITY, **kw).to_host()
    assert ctx.last_variant.startswith("tap pair")
    assert O.rel_err(dx.astype(F), O.conv2d_grad_inputs(w.astype(F), dy.astype(F), (28, 29), **kw)) < tol(dtype)


@DTYPES
@pytest.mark.parametrize("relu", [False, True])
def test_tiles_behind_the_last_whole_wave_are_cut(ctx, dtype, relu):
    """Pair tiles a few more than pairs of SMs; the result of a repeated call is the same bit by bit."""
    c = 256 if dtype == F else 512
    rs = np.random.RandomState(7)
    x = rs.standard_normal((25, c, 28, 28)).astype(dtype)
    w = (rs.standard_normal((128, c, 3, 3)) / np.sqrt(c * 9)).astype(dtype)
    b = rs.standard_normal((1, 128, 1, 1)).astype(dtype)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    call = lambda: shim.device_conv2d(X, W, border_mode="half", bias=B, relu=relu, flags=shim.NO_SLAB).to_host()  # noqa: E731
    y = call()
    assert ctx.last_variant == "tap pair cut"
    assert np.array_equal(y, call())
    part = slice(20, 25)                           # the images of the cut tiles are the last ones
    ref = O.conv2d(x[part].astype(F), w.astype(F), border_mode="half") + b.astype(F)
    assert O.rel_err(y[part].astype(F), np.maximum(ref, 0) if relu else ref) < tol(dtype)
    ctx.set_pair_kernels(False)
    assert O.rel_err(y.astype(F), call().astype(F)) < (1e-5 if dtype == F else 1e-3)


# sides that tiles divide and that they do not, tiles of several images, filters off the tile width, a cut launch, more tiles than images
@DTYPES
@pytest.mark.parametrize("n,h,w_,c,k", [(61, 14, 14, 40, 128), (60, 16, 10, 64, 192), (25, 28, 28, 512, 128), (9, 34, 30, 33, 320), (90, 6, 70, 64, 256)])
def test_pooling(ctx, tmp_path, dtype, n, h, w_, c, k):
    rs = np.random.RandomState(n)
    x = rs.standard_normal((n, c, h, w_)).astype(dtype)
    w = (rs.standard_normal((k, c, 3, 3)) / np.sqrt(c * 9)).astype(dtype)
    b = rs.standard_normal((1, k, 1, 1)).astype(dtype)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    call = lambda pool: shim.device_conv2d(X, W, border_mode="half", bias=B, relu=True, pool=pool)  # noqa: E731
    ctx.set_autotune(True)
    call(True)
    path = str(tmp_path / "t")
    ctx.tuning_save(path)
    head, *rest = open(path).read().splitlines()
    open(path, "w").write("\n".join([head] + [" ".join(r.split()[:2] + ["5"]) if r.startswith("a 3.") else r for r in rest]) + "\n")
    ctx.tuning_load(path)
    y = call(True).to_host().astype(F)
    assert ctx.last_variant == ("tap pair cut" if n == 25 else ctx.last_variant) and ctx.last_variant.startswith("tap pair")
    ctx.set_autotune(False)
    full = call(False).to_host().astype(F)[:, :, :h // 2 * 2, :w_ // 2 * 2]
    ref = full.reshape(n, k, h // 2, 2, w_ // 2, 2).max(axis=(3, 5))
    assert O.rel_err(y, ref) < (1e-5 if dtype == F else 1e-3)      # the same products, sums in another order
