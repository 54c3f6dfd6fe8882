"""gradWeights of tensors with infinities and NaN: whichever kernel runs, an element of the gradient is NaN or infinite where its
own sum is.  The kernels' tiles reach over the images' borders, where zeros stand for dy and x holds real pixels, and zero times
an infinity is NaN."""
import numpy as np
import pytest

from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
T = shim.DeviceTensor


def _gradient(x, dy, ks, pad, s, d, g, flip):
    """The gradient in float64 from the sums themselves; pixels of x outside of the image are zeros that take part."""
    x, dy = x.astype(np.float64), dy.astype(np.float64)
    xp = np.pad(x, ((0, 0), (0, 0), (pad[0], ks * d), (pad[1], ks * d)))
    (n, k, ho, wo), c = dy.shape, x.shape[1] // g
    dw = np.zeros((k, c, ks, ks))
    with np.errstate(invalid="ignore"):
        for i in range(ks):
            for j in range(ks):
                xs = xp[:, :, i * d:i * d + (ho - 1) * s + 1:s, j * d:j * d + (wo - 1) * s + 1:s]
                at = (ks - 1 - i, ks - 1 - j) if flip else (i, j)
                for q in range(g):
                    a, b = dy[:, q * (k // g):(q + 1) * (k // g)], xs[:, q * c:(q + 1) * c]
                    dw[q * (k // g):(q + 1) * (k // g), :, at[0], at[1]] = np.einsum("nkhw,nchw->kc", a, b)
    return dw


def _places(h, w):
    return [(0, w // 2), (h - 1, w // 2), (h // 2, 0), (h // 2, w - 1), (0, 0), (h - 1, w - 1), (h // 2, w // 2)]


# xs, k, ks, stride, dilation, groups, flags, kernel (None: whatever it is)
CASES = {
    "tap": ((3, 20, 13, 11), 24, 3, 1, 1, 1, shim.NO_GROUP, "wgrad tap"),
    "tap-stride": ((3, 20, 13, 17), 140, 3, 2, 1, 1, shim.NO_GROUP, "wgrad tap"),
    "tap-atomic": ((3, 20, 13, 11), 24, 3, 1, 1, 1, shim.NO_GROUP | shim.ATOMIC_SPLITK, "wgrad tap"),
    "pair": ((2, 256, 7, 9), 256, 3, 1, 1, 1, shim.NO_GROUP, "wgrad pair"),
    "groups": ((3, 70, 13, 11), 24, 3, 1, 1, 1, shim.NO_ROWS, "wgrad groups"),
    "groups-wide-image": ((1, 40, 5, 150), 130, 3, 1, 1, 1, 0, "wgrad groups"),
    "groups-stride": ((3, 20, 13, 17), 140, 3, 2, 1, 1, 0, "wgrad groups"),
    "rows": ((3, 20, 13, 11), 24, 3, 1, 1, 1, shim.ROWS, "wgrad rows"),
    "rows-stride": ((3, 20, 14, 17), 24, 3, 2, 1, 1, shim.ROWS, "wgrad rows"),
    "rows-dilation": ((3, 36, 14, 17), 9, 3, 1, 2, 1, shim.ROWS, "wgrad rows"),
    "rows-4x4": ((2, 20, 19, 8), 30, 4, 1, 1, 1, shim.ROWS, "wgrad rows"),
    "merged-rows": ((3, 64, 10, 12), 64, 3, 1, 1, 8, shim.ROWS, "wgrad rows"),
    "merged": ((3, 64, 10, 12), 64, 3, 1, 1, 8, shim.NO_ROWS, "wgrad groups"),
    "two-groups": ((3, 64, 10, 12), 160, 3, 1, 1, 2, shim.NO_GROUP, "wgrad tap"),
    "folded-rows": ((3, 3, 13, 11), 24, 3, 1, 1, 1, shim.ROWS, "wgrad rows"),
    "folded": ((3, 3, 13, 11), 24, 3, 1, 1, 1, shim.NO_ROWS, "wgrad tap"),
    "folded-groups": ((3, 4, 13, 11), 8, 3, 1, 1, 4, 0, None),
    "blocks-rows": ((3, 3, 15, 18), 24, 7, 2, 1, 1, shim.ROWS, "wgrad rows"),
    "blocks": ((3, 3, 15, 18), 24, 7, 2, 1, 1, shim.NO_ROWS, "wgrad tap"),
    "1x1": ((3, 20, 6, 7), 24, 1, 1, 1, 1, 0, None),
}


@DTYPES
@pytest.mark.parametrize("border,flip", [("half", True), ("half", False), ("valid", True), ("full", True)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_sums_are_infinite_or_nan_where_their_products_are(dtype, name, border, flip):
    xs, k, ks, s, d, g, flags, kernel = CASES[name]
    pad = ({"half": ((ks - 1) * d + 1) // 2, "valid": 0, "full": (ks - 1) * d}[border],) * 2
    kw = dict(border_mode=border, subsample=(s, s), filter_dilation=(d, d), num_groups=g, filter_flip=flip)
    ho, wo = ((v + 2 * pad[0] - (ks - 1) * d - 1) // s + 1 for v in xs[2:])
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    rs = np.random.RandomState(len(name))
    odd = lambda shape: (2 * rs.randint(0, 2, shape) - 1).astype(dtype)  # noqa: E731  (-1 and 1: no sum is NaN for a zero factor)
    for where in range(7):
        for layout in ("nhwc", "nchw"):
            special = (np.inf, np.nan, -np.inf)[(where + (layout == "nchw")) % 3]
            x, dy = odd(xs), odd((xs[0], k, ho, wo))
            if where % 2:
                dy[:] *= rs.randint(0, 2, dy.shape).astype(dtype)           # with zeros, whose product with an infinity is NaN
            r, q = _places(*xs[2:])[where]
            x[rs.randint(xs[0]), rs.randint(xs[1]), r, q] = special
            if special == -np.inf:
                r, q = _places(ho, wo)[where]
                dy[rs.randint(xs[0]), rs.randint(k), r, q] = special
            got = shim.device_grad_weights(T.from_host(ctx, x, layout), T.from_host(ctx, dy, layout), (ks, ks), flags=flags, **kw).to_host()
            assert np.array_equal(got.astype(np.float64), _gradient(x, dy, ks, pad, s, d, g, flip), equal_nan=True), (layout, special, where)
            assert ctx.last_variant == kernel or kernel is None
    ctx.close()


@pytest.mark.parametrize("name", ["rows", "merged-rows", "folded-rows", "blocks-rows", "tap"])
def test_float32_gradients_of_float16_tensors_in_a_graph(name):
    xs, k, ks, s, d, g, flags, kernel = CASES[name]
    pad = (((ks - 1) * d + 1) // 2,) * 2
    kw = dict(border_mode="half", subsample=(s, s), num_groups=g)
    ho, wo = ((v + 2 * pad[0] - ks) // s + 1 for v in xs[2:])
    ctx = shim.Context(0)
    rs = np.random.RandomState(3)
    x, dy = (2 * rs.randint(0, 2, v) - 1.0 for v in (xs, (xs[0], k, ho, wo)))
    x[1, 0, 0, 3], x[0, xs[1] - 1, xs[2] - 1, 2], dy[2, 1, ho // 2, 0] = np.inf, np.nan, -np.inf
    X, DY = T.from_host(ctx, x.astype(np.float16), "nhwc"), T.from_host(ctx, dy.astype(np.float16), "nhwc")
    DW = T(ctx, (k, xs[1] // g, ks, ks), np.float32)
    run = lambda: shim.device_grad_weights(X, DY, (ks, ks), out=DW, flags=flags, **kw)  # noqa: E731
    run()
    graph = ctx.capture(run)
    ctx.memset(DW.ptr, 0, DW.nbytes)
    graph.launch()
    assert np.array_equal(DW.to_host().astype(np.float64), _gradient(x, dy, ks, pad, s, 1, g, True), equal_nan=True)
    assert ctx.last_variant == kernel
    graph.destroy()
    ctx.close()


@DTYPES
def test_finite_sums_among_infinite_ones_are_exact(dtype):
    """Sums taken again are those of the definition: against float64, real values, many images."""
    ctx = shim.Context(0)
    rs = np.random.RandomState(5)
    x, dy = rs.standard_normal((40, 16, 14, 14)).astype(dtype), rs.standard_normal((40, 16, 14, 14)).astype(dtype)
    x[7, :, 0, :] = np.inf                               # the whole first row: every channel's filter row that stays off it
    want = _gradient(x, dy, 3, (1, 1), 1, 1, 1, True)
    got = shim.device_grad_weights(T.from_host(ctx, x, "nhwc"), T.from_host(ctx, dy, "nhwc"), (3, 3), border_mode="half", flags=shim.ROWS).to_host()
    finite = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), finite) and finite.sum() == 16 * 16 * 3
    # float32: summed in double, rounded once; float16: the result's rounding
    assert np.allclose(got[finite].astype(np.float64), want[finite], rtol=1e-6 if dtype == np.float32 else 1e-3, atol=1e-6)
    ctx.close()
