"""The columns kernel: filter widths that fill the pitches of 8, 16 and 32 positions, images that end inside tiles and rows, filter
counts with rows of 32, 64 and 128 bytes, groups, dilation, both directions, pooling, and infinities in the input."""
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
    yield c
    c.close()


def tol(dtype):
    return 5e-3 if dtype == F else 2e-2            # the repository's bounds for TF32 factors and float16 tensors


def columns_only(ctx, path, call, pair=False):
    """Makes the remembered choice of every geometry that `call` meets the columns kernel (on pairs of CTAs), then runs it."""
    call()
    ctx.tuning_save(path)
    head, *rest = open(path).read().splitlines()
    open(path, "w").write("\n".join([head] + [" ".join(r.split()[:2] + ["7" if pair else "6"]) if r.startswith("a 3.") else r for r in rest]) + "\n")
    ctx.tuning_load(path)
    y = call()
    assert ctx.last_variant == ("columns pair" if pair else "columns")
    return y


# images, height, width, channels, filters, kernel, dilation, groups
LAYERS = [(2, 13, 30, 48, 32, (3, 3), 1, 1), (1, 9, 31, 24, 64, (3, 3), 1, 1), (3, 14, 14, 64, 16, (3, 3), 1, 1), (2, 7, 6, 40, 24, (3, 3), 1, 1),
          (2, 28, 28, 128, 128, (3, 3), 1, 4), (1, 40, 45, 33, 12, (1, 5), 1, 1), (2, 19, 37, 70, 48, (5, 2), 2, 1), (1, 33, 17, 16, 8, (4, 8), 1, 1),
          (1, 64, 50, 12, 30, (7, 7), 1, 1), (2, 20, 24, 96, 64, (2, 4), 3, 1), (150, 16, 16, 64, 64, (3, 3), 1, 2)]


@DTYPES
@pytest.mark.parametrize("n,h,w_,c,k,ks,d,g", LAYERS)
def test_forward_against_the_oracle(ctx, tmp_path, dtype, n, h, w_, c, k, ks, d, g):
    rs = np.random.RandomState(n + k)
    kw = dict(border_mode="half", filter_dilation=(d, d), num_groups=g)
    x = rs.standard_normal((n, c, h, w_)).astype(dtype)
    w = (rs.standard_normal((k, c // g) + ks) / np.sqrt(c // g * ks[0] * ks[1])).astype(dtype)
    b = rs.standard_normal((1, k, 1, 1)).astype(dtype)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    y = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, bias=B, relu=True, **kw))
    ref = np.maximum(O.conv2d(x.astype(F), w.astype(F), **kw) + b.astype(F), 0)
    assert O.rel_err(y.to_host().astype(F), ref) < tol(dtype)


@DTYPES
@pytest.mark.parametrize("n,h,w_,c,k,ks,d,g", [(2, 13, 30, 32, 40, (3, 3), 1, 1), (1, 24, 33, 60, 70, (5, 3), 2, 1), (2, 28, 28, 128, 128, (3, 3), 1, 4)])
def test_grad_inputs_against_the_oracle(ctx, tmp_path, dtype, n, h, w_, c, k, ks, d, g):
    rs = np.random.RandomState(n + k)
    kw = dict(border_mode="half", filter_dilation=(d, d), num_groups=g)
    w = (rs.standard_normal((k, c // g) + ks) / np.sqrt(k // g * ks[0] * ks[1])).astype(dtype)
    dy = rs.standard_normal((n, k, h, w_)).astype(dtype)
    W, DY = T.from_host(ctx, w), T.from_host(ctx, dy, "nhwc")
    dx = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_grad_inputs(W, DY, (h, w_), **kw))
    assert O.rel_err(dx.to_host().astype(F), O.conv2d_grad_inputs(w.astype(F), dy.astype(F), (h, w_), **kw)) < tol(dtype)


# odd numbers of tiles, more and fewer than pairs of SMs, filters between 33 and 64
PAIRS = [(1, 9, 31, 24, 64, (3, 3), 1, 1), (3, 14, 14, 64, 40, (3, 3), 1, 1), (1, 200, 61, 33, 48, (1, 4), 1, 1), (5, 61, 61, 70, 64, (5, 2), 2, 1),
         (150, 16, 16, 128, 128, (3, 3), 1, 2), (33, 56, 28, 130, 64, (3, 3), 1, 1)]


@DTYPES
@pytest.mark.parametrize("n,h,w_,c,k,ks,d,g", PAIRS)
def test_pairs_against_the_oracle(ctx, tmp_path, dtype, n, h, w_, c, k, ks, d, g):
    rs = np.random.RandomState(n + k)
    kw = dict(border_mode="half", filter_dilation=(d, d), num_groups=g)
    x = rs.standard_normal((n, c, h, w_)).astype(dtype)
    w = (rs.standard_normal((k, c // g) + ks) / np.sqrt(c // g * ks[0] * ks[1])).astype(dtype)
    b = rs.standard_normal((1, k, 1, 1)).astype(dtype)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    y = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, bias=B, relu=True, **kw), pair=True)
    ref = np.maximum(O.conv2d(x.astype(F), w.astype(F), **kw) + b.astype(F), 0)
    assert O.rel_err(y.to_host().astype(F), ref) < tol(dtype)
    one = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, bias=B, relu=True, **kw))
    assert np.array_equal(y.to_host(), one.to_host())      # the same sums


# filters that stay for all tiles of a CTA (several per CTA): one and more channel blocks, groups that divide the CTAs
# and groups that leave some of them out, and numbers of blocks that do not fit
STAY = [(40, 24, 64, 1), (40, 64, 64, 1), (40, 128, 64, 1), (40, 100, 36, 1), (40, 130, 64, 1), (20, 128, 128, 2), (6, 512, 512, 8), (6, 256, 256, 8),
        (3, 96, 96, 3), (40, 256, 57, 1)]


@DTYPES
@pytest.mark.parametrize("n,c,k,g,pair", [a + (p,) for a in STAY for p in (False, True) if not p or a[2] // a[3] > 32])
def test_filters_that_stay(ctx, tmp_path, dtype, n, c, k, g, pair):
    rs = np.random.RandomState(k)
    kw = dict(border_mode="half", num_groups=g)
    x = rs.standard_normal((n, c, 56, 54)).astype(dtype)
    w = (rs.standard_normal((k, c // g, 3, 3)) / np.sqrt(9 * c // g)).astype(dtype)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    y = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, **kw), pair=pair)
    some = [0, n // 2, n - 1]
    ref = O.conv2d(x[some].astype(F), w.astype(F), **kw)
    assert O.rel_err(y.to_host()[some].astype(F), ref) < tol(dtype)


@DTYPES
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("n,h,w_,c,k", [(2, 28, 30, 24, 64), (3, 10, 62, 40, 64), (40, 56, 56, 24, 64)])
def test_pooling(ctx, tmp_path, dtype, n, h, w_, c, k, pair):
    rs = np.random.RandomState(n)
    x = rs.standard_normal((n, c, h, w_)).astype(dtype)
    w = (rs.standard_normal((k, c, 3, 3)) / np.sqrt(c * 9)).astype(dtype)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    y = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, border_mode="half", relu=True, pool=True), pair)
    full = shim.device_conv2d(X, W, border_mode="half", relu=True).to_host().astype(F)
    ref = full.reshape(n, k, h // 2, 2, w_ // 2, 2).max(axis=(3, 5))
    assert O.rel_err(y.to_host().astype(F), ref) < (1e-5 if dtype == F else 1e-3)      # the same products, sums in another order


@DTYPES
def test_an_infinity_stays_with_the_outputs_that_it_belongs_to(ctx, tmp_path, dtype):
    rs = np.random.RandomState(1)
    x = rs.standard_normal((2, 20, 17, 29)).astype(dtype)
    x[1, 3, 8, 28] = np.inf
    w = (1 + rs.random_sample((30, 20, 3, 3))).astype(dtype)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    y = columns_only(ctx, str(tmp_path / "t"), lambda: shim.device_conv2d(X, W, border_mode="half")).to_host()
    touched = np.zeros(y.shape, bool)
    touched[1, :, 7:10, 27:29] = True
    assert np.array_equal(~np.isfinite(y), touched)
    stored = np.empty((2, 17, 29, ctx.padded_channels(30, dtype)), dtype)
    Y = shim.device_conv2d(X, W, border_mode="half")
    ctx.d2h(stored, Y.ptr)
    ctx.sync()
    assert not stored[..., 30:].any()


@DTYPES
@pytest.mark.parametrize("h,ks,d", [(150, (3, 3), (128, 1)), (260, (2, 4), (256, 2)), (40, (5, 3), (64, 1)), (150, (3, 2), (127, 1))])
def test_filters_that_reach_over_256_rows(ctx, dtype, h, ks, d):
    """Dilated filters of a box's 256 rows and about: no tile of the columns kernel holds them, the layer runs on another."""
    rs = np.random.RandomState(h)
    kw = dict(border_mode="half", filter_dilation=d)
    x = rs.standard_normal((2, 20, h, 17)).astype(dtype)
    w = (rs.standard_normal((24, 20) + ks) / np.sqrt(20 * ks[0] * ks[1])).astype(dtype)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    ref = O.conv2d(x.astype(F), w.astype(F), **kw)
    y = shim.device_conv2d(X, W, **kw)
    assert not ctx.last_variant.startswith("columns")
    assert O.rel_err(y.to_host().astype(F), ref) < tol(dtype)
    dy = rs.standard_normal(ref.shape).astype(dtype)
    dx = shim.device_grad_inputs(W, T.from_host(ctx, dy, "nhwc"), (h, 17), **kw)
    assert not ctx.last_variant.startswith("columns")
    assert O.rel_err(dx.to_host().astype(F), O.conv2d_grad_inputs(w.astype(F), dy.astype(F), (h, 17), **kw)) < tol(dtype)
