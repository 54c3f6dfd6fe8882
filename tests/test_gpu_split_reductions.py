"""Forward and gradInputs of few output tiles (narrow tiles, reductions split over CTAs), the pad channels of
channels-last outputs, and tensors that start off the 16-byte boundaries."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
TOL = {np.float32: 5e-3, np.float16: 2e-2}      # the repository's bounds: TF32 factors, float16 tensors


@pytest.fixture
def ctx():
    """A context that takes the model's choice of kernel, which is the spread variant wherever there is one."""
    c = shim.Context(0)
    c.set_autotune(False)
    yield c
    c.close()


def stored(t):
    """A channels-last tensor as it lies in memory, pad channels included."""
    n, _, h, w = t.shape
    a = np.empty((n, h, w, t.stored_channels), t.dtype)
    t.ctx.d2h(a, t.ptr)
    t.ctx.sync()
    return a


# one or a few images, reductions from one step to 144; filters below, at and above a tile's columns
SPLIT = [((1, 512, 14, 14), 512, 3, 1), ((1, 512, 7, 7), 75, 3, 1), ((2, 33, 9, 5), 20, 5, 1), ((1, 64, 8, 8), 32, 1, 1),
         ((1, 1000, 6, 7), 257, 1, 1), ((3, 130, 13, 11), 129, 3, 2), ((1, 8, 3, 3), 5, 3, 1), ((1, 2048, 1, 1), 64, 1, 1)]


@DTYPES
@pytest.mark.parametrize("flags", [0, shim.NO_SLAB], ids=["slab", "tap"])
@pytest.mark.parametrize("xs,k,ks,s", SPLIT, ids=lambda v: str(v).replace(" ", ""))
def test_split_reductions_against_oracle(ctx, dtype, flags, xs, k, ks, s):
    rs = np.random.RandomState(k)
    x = rs.standard_normal(xs).astype(dtype)
    w = (rs.standard_normal((k, xs[1], ks, ks)) / np.sqrt(xs[1] * ks * ks)).astype(dtype)
    b = rs.standard_normal(k).astype(dtype)
    kw = dict(border_mode="half", subsample=(s, s))
    f = np.float32
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b.reshape(1, k, 1, 1))
    conv = O.conv2d(x.astype(f), w.astype(f), **kw)
    dy = rs.standard_normal(conv.shape).astype(dtype)
    R = DY = T.from_host(ctx, dy, "nhwc")
    y = shim.device_conv2d(X, W, bias=B, residual=R, relu=True, slope=0.1, alpha=0.5, beta=2., flags=flags, **kw)
    v = 0.5 * conv + b.astype(f)[None, :, None, None] + 2 * dy.astype(f)
    assert O.rel_err(y.to_host().astype(f), np.where(v > 0, v, 0.1 * v)) < TOL[dtype]
    assert not stored(y)[..., k:].any()
    dx = shim.device_grad_inputs(W, DY, xs[2:], flags=flags, **kw)
    assert O.rel_err(dx.to_host().astype(f), O.conv2d_grad_inputs(w.astype(f), dy.astype(f), xs[2:], **kw)) < TOL[dtype]
    assert not stored(dx)[..., xs[1]:].any()
    y = shim.device_conv2d(X, W, out_layout="nchw", flags=flags, **kw)
    assert O.rel_err(y.to_host().astype(f), conv) < TOL[dtype]


@DTYPES
@pytest.mark.parametrize("flags", [0, shim.NO_SLAB], ids=["slab", "tap"])
@pytest.mark.parametrize("xs,k,ks", [((1, 512, 8, 8), 75, 3),       # split reduction
                                     ((40, 16, 28, 28), 62, 3),     # whole 128-byte channel chunks in float32
                                     ((40, 16, 28, 28), 21, 3),     # direct stores
                                     ((16, 256, 40, 40), 255, 1)],  # pairs of CTAs in float16
                         ids=["split", "staged", "direct", "pair"])
def test_infinities_leave_pad_channels_zero(ctx, dtype, flags, xs, k, ks):
    """Pad channels are the product of zero filters and the input; an infinity there would make them NaN."""
    rs = np.random.RandomState(5)
    x = rs.standard_normal(xs).astype(dtype)
    x[0, 1, 3, 2] = np.inf
    w = (rs.standard_normal((k, xs[1], ks, ks)) / np.sqrt(xs[1] * ks * ks)).astype(dtype)
    y = shim.device_conv2d(T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), border_mode="half", flags=flags)
    a = stored(y)
    assert a.shape[-1] > k and not a[..., k:].any()
    assert np.isinf(a[0, 3, 2, :k]).all() and np.isfinite(a[1:]).all()
    # gradInputs of the mirrored layer: its input has the k (padded) channels
    dx = shim.device_grad_inputs(T.from_host(ctx, np.ascontiguousarray(w.transpose(1, 0, 2, 3))), T.from_host(ctx, x, "nhwc"),
                                 xs[2:], border_mode="half", flags=flags)
    a = stored(dx)
    assert not a[..., k:].any() and np.isinf(a[0, 3, 2, :k]).all() and np.isfinite(a[1:]).all()


def shifted(t, fill=None):
    """The same tensor in memory one element off the 16-byte boundaries (and the memory's owner)."""
    es = t.dtype.itemsize
    owner = T(t.ctx, (1, 1, 1, t.nbytes // es + 16), t.dtype)
    view = T(t.ctx, t.shape, t.dtype, t.layout, _ptr=owner.ptr + es)
    a = stored(t) if fill is None else np.full((t.nbytes // es,), fill, t.dtype)
    t.ctx.h2d(view.ptr, a)
    t.ctx.sync()
    return view, owner


@DTYPES
@pytest.mark.parametrize("shape", [(2, 33, 9, 6), (1, 8, 5, 5)], ids=["33ch", "8ch"])
def test_pooling_and_channel_sum_off_the_boundary(ctx, dtype, shape):
    rs = np.random.RandomState(3)
    n, c, h, w = shape
    x = rs.standard_normal(shape).astype(dtype)
    X = T.from_host(ctx, x, "nhwc")
    Y = shim.device_maxpool2x2(X)
    G = T.from_host(ctx, rs.standard_normal(Y.shape).astype(dtype), "nhwc")
    GX = shim.device_maxpool2x2_grad(X, Y, G)
    (Xs, o1), (Ys, o2), (Gs, o3), (GXs, o4) = shifted(X), shifted(Y, 7), shifted(G), shifted(GX, 7)
    assert np.array_equal(stored(shim.device_maxpool2x2(Xs, out=Ys)), stored(Y))
    assert np.array_equal(stored(shim.device_maxpool2x2_grad(Xs, Ys, Gs, out=GXs)), stored(GX))
    # float32 sums of at most 108 values of order 1 in another order; float16 results round to 2^-11 on top
    want = x.astype(np.float64).sum((0, 2, 3))
    tol = 1e-4 if dtype == np.float32 else 2e-2
    assert np.abs(shim.device_channel_sum(Xs) - want).max() < tol and np.abs(shim.device_channel_sum(X) - want).max() < tol


@DTYPES
@pytest.mark.parametrize("flags", [0, shim.NO_SLAB], ids=["slab", "tap"])
@pytest.mark.parametrize("xs,k", [((1, 512, 8, 8), 75), ((40, 16, 28, 28), 21), ((40, 16, 28, 28), 64)], ids=["split", "direct", "whole"])
def test_outputs_off_the_boundary(ctx, dtype, flags, xs, k):
    rs = np.random.RandomState(4)
    X = T.from_host(ctx, rs.standard_normal(xs).astype(dtype), "nhwc")
    W = T.from_host(ctx, (rs.standard_normal((k, xs[1], 3, 3)) / np.sqrt(xs[1] * 9)).astype(dtype))
    y = shim.device_conv2d(X, W, border_mode="half", flags=flags)
    ys, owner = shifted(y, 7)
    shim.device_conv2d(X, W, border_mode="half", out=ys, flags=flags)
    a, b = stored(y).astype(np.float32), stored(ys).astype(np.float32)
    assert O.rel_err(b, a) < TOL[dtype] / 4          # another tile may split the sums elsewhere


@DTYPES
def test_pooling_epilogue_still_asks_for_whole_channel_chunks(ctx, dtype):
    """A split reduction could pool any channel count, but what the epilogue refuses does not depend on the batch."""
    X = T.from_host(ctx, np.ones((1, 512, 8, 8), dtype), "nhwc")
    W = T.from_host(ctx, np.ones((75, 512, 3, 3), dtype))
    with pytest.raises(shim.B200Error, match="cannot pool"):
        shim.device_conv2d(X, W, border_mode="half", pool=True)


@DTYPES
def test_what_the_epilogue_refuses_does_not_depend_on_earlier_calls(dtype):
    """An output off the 16-byte boundaries is refused also when an aligned one has chosen a split reduction before."""
    own = shim.Context(0)                        # with timing
    X = T.from_host(own, np.ones((1, 512, 8, 8), dtype), "nhwc")
    W = T.from_host(own, np.ones((64, 512, 3, 3), dtype))
    y = shim.device_conv2d(X, W, border_mode="half", pool=True)
    ys, owner = shifted(y, 7)
    for _ in range(2):
        with pytest.raises(shim.B200Error, match="cannot pool"):
            shim.device_conv2d(X, W, border_mode="half", pool=True, out=ys)
        assert (stored(ys) == 7).all()
        shim.device_conv2d(X, W, border_mode="half", pool=True, out=y)
    own.close()


@DTYPES
@pytest.mark.parametrize("c,k,g", [(256, 256, 32), (96, 48, 12), (64, 128, 8), (48, 48, 3), (512, 256, 2)], ids=lambda v: str(v))
def test_grad_weights_of_merged_groups(ctx, dtype, c, k, g):
    rs = np.random.RandomState(g)
    x, dy = (rs.standard_normal((3, n, 11, 9)).astype(dtype) for n in (c, k))
    kw = dict(border_mode="half", num_groups=g)
    dw = shim.device_grad_weights(T.from_host(ctx, x, "nhwc"), T.from_host(ctx, dy, "nhwc"), (3, 3), **kw).to_host()
    f = np.float32
    assert O.rel_err(dw.astype(f), O.conv2d_grad_weights(x.astype(f), dy.astype(f), (3, 3), **kw)) < TOL[dtype]


@DTYPES
@pytest.mark.parametrize("shape", [(2, 33, 9, 6), (3, 8, 41, 31), (1, 5, 1, 1)], ids=["33ch", "8ch", "one"])
def test_elementwise_off_the_boundary(ctx, dtype, shape):
    """Any of the three tensors may start off the 16-byte boundaries; the results are those of aligned tensors."""
    rs = np.random.RandomState(7)
    A, B = (T.from_host(ctx, rs.standard_normal(shape).astype(dtype), "nhwc") for _ in range(2))
    (As, o1), (Bs, o2) = shifted(A), shifted(B)
    v = rs.standard_normal(shape[1]).astype(dtype)
    for op, aligned, off in (("add", B, Bs), ("mul", 0.5, 0.5), ("sub", v, v), ("sgn", None, None)):
        want = stored(shim.device_elementwise(op, A, aligned))
        for a in (A, As):
            for b in {id(aligned): aligned, id(off): off}.values():
                for make in (lambda: (T(ctx, shape, dtype, "nhwc"), None), lambda: shifted(A, 7)):
                    out, owner = make()
                    assert np.array_equal(stored(shim.device_elementwise(op, a, b, out=out)), want), (op, a is As, owner)
    out, owner = shifted(A)
    assert np.array_equal(stored(shim.device_elementwise("add", out, Bs, out=out)), stored(shim.device_elementwise("add", A, B)))


# few-channel layers, whose images are rearranged first: folded rows and 2x2 pixel blocks; strided gradInputs whose
# parity classes are channels of one launch
STEMS = [((2, 3, 20, 17), 24, 3, 1), ((3, 1, 15, 18), 8, 5, 1), ((2, 3, 21, 22), 64, 7, 2), ((2, 4, 16, 16), 16, 3, 2)]


@DTYPES
@pytest.mark.parametrize("xs,k,ks,s", STEMS, ids=lambda v: str(v).replace(" ", ""))
def test_stems_off_the_boundary(ctx, dtype, xs, k, ks, s):
    rs = np.random.RandomState(8)
    X = T.from_host(ctx, rs.standard_normal(xs).astype(dtype), "nhwc")
    W = T.from_host(ctx, (rs.standard_normal((k, xs[1], ks, ks)) / ks).astype(dtype))
    Xs, owner = shifted(X)
    kw = dict(border_mode="half", subsample=(s, s))
    Y = shim.device_conv2d(X, W, **kw)
    assert np.array_equal(stored(shim.device_conv2d(Xs, W, **kw)), stored(Y))
    DY = T.from_host(ctx, rs.standard_normal(Y.shape).astype(dtype), "nhwc")
    assert np.array_equal(shim.device_grad_weights(Xs, DY, (ks, ks), **kw).to_host(),
                          shim.device_grad_weights(X, DY, (ks, ks), **kw).to_host())
    if s > 1:
        DX = shim.device_grad_inputs(W, DY, xs[2:], **kw)
        DXs, owner2 = shifted(X, 7)
        assert np.array_equal(stored(shim.device_grad_inputs(W, DY, xs[2:], out=DXs, **kw)), stored(DX))
        assert not stored(DXs)[..., xs[1]:].any()


def test_split_reductions_fall_back_to_whole_ones_without_memory_for_slices():
    """A 1x1 forward call on channels-last tensors needs no scratch but the slices of a split reduction (4 MB and more
    here); with the device's memory taken, it runs unsplit."""
    rs = np.random.RandomState(9)
    x = rs.standard_normal((1, 2048, 14, 14)).astype(np.float32)
    w = (rs.standard_normal((512, 2048, 1, 1)) / 45).astype(np.float32)
    c = shim.Context(0)
    c.set_autotune(False)
    c.set_pair_kernels(False)
    # the kernels' code is on the device before its memory is taken: split and whole, with both kernels
    many = T(c, (64, 2048, 14, 14), np.float32, "nhwc")
    W = T.from_host(c, w)
    for flags in (0, shim.NO_SLAB):
        for X in (T.from_host(c, x, "nhwc"), many):
            shim.device_conv2d(X, W, flags=flags)
    c.sync()
    c.close()
    c = shim.Context(0)
    c.set_autotune(False)
    c.set_pair_kernels(False)
    X, W, Y = T.from_host(c, x, "nhwc"), T.from_host(c, w), T(c, (1, 512, 14, 14), np.float32, "nhwc")
    want = O.conv2d(x, w)
    taken, size = [], 256 << 30
    while size >= 2 << 20:
        try:
            taken.append(T(c, (1, 1, 1, size // 4), np.float32))
        except (MemoryError, shim.B200Error):
            size //= 2
    try:
        free = c.memory_info()[1]
        assert free < 4 << 20, free
        for flags in (0, shim.NO_SLAB):
            before = c.launches
            shim.device_conv2d(X, W, out=Y, flags=flags)
            assert c.launches - before == 1                              # no second kernel that adds slices
        c.sync()
    finally:
        for t in taken:
            t.free()
    assert O.rel_err(Y.to_host(), want) < 5e-3
    before = c.launches
    shim.device_conv2d(X, W, out=Y)
    assert c.launches - before == 2                                      # with memory again: split
    c.close()


@DTYPES
@pytest.mark.parametrize("flags", [0, shim.NO_SLAB], ids=["slab", "tap"])
@pytest.mark.parametrize("xs,k,ks", [((1, 512, 8, 8), 75, 3), ((40, 16, 28, 28), 21, 3), ((16, 256, 40, 40), 255, 1)], ids=["split", "direct", "1x1"])
def test_pad_channels_of_a_residual_stay_out_of_the_result(ctx, dtype, flags, xs, k, ks):
    """Pad channels are written as zeros whatever the pad channels of the residual hold, also off the 16-byte boundaries."""
    rs = np.random.RandomState(10)
    x = rs.standard_normal(xs).astype(dtype)
    w = (rs.standard_normal((k, xs[1], ks, ks)) / np.sqrt(xs[1] * ks * ks)).astype(dtype)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    conv = O.conv2d(x.astype(np.float32), w.astype(np.float32), border_mode="half", subsample=(1, 1))
    r = rs.standard_normal(conv.shape).astype(dtype)
    R = T.from_host(ctx, r, "nhwc")
    a = stored(R)
    a[..., k:] = np.nan
    ctx.h2d(R.ptr, a)
    out = T(ctx, conv.shape, dtype, "nhwc")
    off, owner = shifted(out, 7)
    for y in (out, off, R):                     # the last one accumulates in place
        shim.device_conv2d(X, W, border_mode="half", residual=R, out=y, flags=flags)
        assert not stored(y)[..., k:].any()
        assert O.rel_err(y.to_host().astype(np.float32), conv + r.astype(np.float32)) < TOL[dtype]
