"""The memory-bound kernels at the edges of their tiles: filter packing and the split-K reduction over tap
counts, pooling, element-wise ops and the per-channel sum over channel counts and odd sizes."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


def upload(ctx, a):
    return shim.DeviceTensor.from_host(ctx, a, "nhwc")


@DTYPES
@pytest.mark.parametrize("kh,kw", [(1, 1), (1, 2), (3, 3), (5, 5), (7, 7), (8, 8)])
@pytest.mark.parametrize("c,k", [(9, 5), (33, 40), (70, 129)])
def test_packing_and_reduction_over_tap_counts(dtype, kh, kw, c, k):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(kh * 100 + c)
    x = rs.standard_normal((2, c, 13, 11)).astype(dtype)
    w = (rs.standard_normal((k, c, kh, kw)) / np.sqrt(c * kh * kw)).astype(dtype)
    kw_ = dict(border_mode="half", subsample=(1, 1))
    X, W = upload(ctx, x), shim.DeviceTensor.from_host(ctx, w)
    y = shim.device_conv2d(X, W, **kw_)
    dy = rs.standard_normal(y.shape).astype(dtype)
    DY = upload(ctx, dy)
    f = np.float32
    # the repository's bounds: 5e-3 of the largest result with TF32 factors, 2e-2 with float16 tensors
    tol = 5e-3 if dtype == np.float32 else 2e-2
    assert O.rel_err(y.to_host().astype(f), O.conv2d(x.astype(f), w.astype(f), **kw_)) < tol
    dx = shim.device_grad_inputs(W, DY, x.shape[2:], **kw_).to_host()
    assert O.rel_err(dx.astype(f), O.conv2d_grad_inputs(w.astype(f), dy.astype(f), x.shape[2:], **kw_)) < tol
    dw = shim.device_grad_weights(X, DY, (kh, kw), **kw_).to_host()
    assert O.rel_err(dw.astype(f), O.conv2d_grad_weights(x.astype(f), dy.astype(f), (kh, kw), **kw_)) < tol


@DTYPES
@pytest.mark.parametrize("splits", [1, 2, 5, 9, 33])
def test_reduction_over_slab_counts(dtype, splits):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(splits)
    x, dy = (rs.standard_normal(s).astype(dtype) for s in ((16, 20, 24, 24), (16, 12, 22, 22)))
    X, DY = upload(ctx, x), upload(ctx, dy)
    ctx.set_splits(splits)
    try:
        dw = shim.device_grad_weights(X, DY, (3, 3)).to_host()
    finally:
        ctx.set_splits(0)
    f = np.float32
    ref = O.conv2d_grad_weights(x.astype(f), dy.astype(f), (3, 3), border_mode="valid", subsample=(1, 1))
    assert O.rel_err(dw.astype(f), ref) < (5e-3 if dtype == np.float32 else 2e-2)


@DTYPES
@pytest.mark.parametrize("shape", [(1, 1, 2, 2), (3, 5, 7, 8), (2, 8, 9, 5), (2, 33, 16, 6), (1, 64, 31, 31)])
def test_channels_last_pooling_and_gradient(dtype, shape):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(shape[1])
    n, c, h, w = shape
    x = rs.randint(-3, 4, shape).astype(dtype)              # ties included
    crop = x[:, :, :h // 2 * 2, :w // 2 * 2]
    win = crop.reshape(n, c, h // 2, 2, w // 2, 2)
    y = win.max(axis=(3, 5))
    gy = rs.standard_normal(y.shape).astype(dtype)
    X = upload(ctx, x)
    Y = shim.device_maxpool2x2(X)
    assert np.array_equal(Y.to_host(), y)
    gx = shim.device_maxpool2x2_grad(X, Y, upload(ctx, gy)).to_host()
    ref = np.zeros_like(x)
    ref[:, :, :h // 2 * 2, :w // 2 * 2] = np.where(win == y[:, :, :, None, :, None], gy[:, :, :, None, :, None],
                                                   dtype(0)).reshape(crop.shape)
    assert np.array_equal(gx, ref)


@DTYPES
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 8, 1, 63), (2, 3, 17, 19), (3, 100, 33, 31), (1, 2049, 3, 3)])
def test_elementwise_and_channel_sum(dtype, shape):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(shape[1])
    a, b = rs.standard_normal(shape).astype(dtype), rs.standard_normal(shape).astype(dtype)
    v = rs.standard_normal(shape[1]).astype(dtype)
    A, B = upload(ctx, a), upload(ctx, b)
    f = np.float32
    for out, ref in ((shim.device_elementwise("mul", A, B), a.astype(f) * b.astype(f)),
                     (shim.device_elementwise("add", A, 0.5), a.astype(f) + f(0.5)),
                     (shim.device_elementwise("sub", A, v), a.astype(f) - v.astype(f)[None, :, None, None]),
                     (shim.device_elementwise("sgn", A), np.sign(a.astype(f)))):
        assert np.array_equal(out.to_host(), ref.astype(dtype))
        # pad channels stay zero, so the sum over channels of the stored tensor is that of the real ones
        assert np.array_equal(shim.device_elementwise("abs", out).to_host(), abs(ref.astype(dtype)))
    got, ref = shim.device_channel_sum(A), a.astype(np.float64).sum(axis=(0, 2, 3))
    # float32 sums of n values of size about 1 in chains of at most n: n * 2^-24 * sum of sizes bounds the error;
    # the result is then rounded to the data type
    size = np.abs(a.astype(np.float64)).sum(axis=(0, 2, 3))
    n = shape[0] * shape[2] * shape[3]
    eps = 2.0 ** -24 if dtype == np.float32 else 2.0 ** -11
    assert got.dtype == dtype and np.all(np.abs(got - ref) <= n * 2.0 ** -24 * size + eps * np.abs(ref) + 1e-7)


@DTYPES
@pytest.mark.parametrize("layout", ["nhwc", "nchw", "off"])
@pytest.mark.parametrize("c,kw,d,border", [(1, 3, 1, "half"), (4, 3, 1, "valid"), (5, 3, 1, (1, 2)), (8, 4, 2, "half"), (9, 3, 1, "half"), (12, 2, 1, (2, 3)), (16, 3, 1, "half")])
def test_folded_images_of_one_and_two_pieces_per_pixel(dtype, layout, c, kw, d, border):
    """Few channels: a filter row is one reduction block over a copy of the image; from both layouts, and from channels-last tensors off the 16-byte
    boundaries.  What the pad channels of a channels-last tensor hold does not matter."""
    ctx = shim.get_context(0)
    rs = np.random.RandomState(c * 10 + kw)
    f = np.float32
    c = c if dtype == np.float16 else (c + 1) // 2           # a block is 64 float16 or 32 float32 numbers
    x = rs.standard_normal((3, c, 12, 9)).astype(dtype)
    w = (rs.standard_normal((20, c, 3, kw)) / np.sqrt(c * 3 * kw)).astype(dtype)
    kw_ = dict(border_mode=border, subsample=(1, 1), filter_dilation=(d, 1))
    if layout == "nchw":
        X = shim.DeviceTensor.from_host(ctx, x)
    else:
        cp = ctx.padded_channels(c, dtype)
        stored = np.full((3, 12, 9, cp), np.inf if cp * x.itemsize > 16 else 0, dtype)
        stored[..., :c] = x.transpose(0, 2, 3, 1)
        room = shim.DeviceTensor(ctx, (1, 1, 1, stored.size + 8), dtype)
        X = shim.DeviceTensor(ctx, x.shape, dtype, "nhwc", _ptr=room.ptr + (4 if layout == "off" else 0))
        ctx.h2d(X.ptr, stored)
    ref = O.conv2d(x.astype(f), w.astype(f), **kw_)
    tol = 5e-3 if dtype == f else 2e-2                       # the repository's bounds, as above
    y = shim.device_conv2d(X, shim.DeviceTensor.from_host(ctx, w), out_layout="nhwc", **kw_)
    assert O.rel_err(y.to_host().astype(f), ref) < tol
    dy = rs.standard_normal(ref.shape).astype(dtype)
    dw = shim.device_grad_weights(X, shim.DeviceTensor.from_host(ctx, dy, X.layout), (3, kw), **kw_).to_host()
    assert O.rel_err(dw.astype(f), O.conv2d_grad_weights(x.astype(f), dy.astype(f), (3, kw), **kw_)) < tol
