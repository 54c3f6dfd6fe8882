"""gradWeights with the filter's rows and columns inside one MMA: filters and channels at the edges of the swizzle atoms,
filter shapes that give one to four sets of rows, strides, dilations, groups, images smaller and larger than a tile."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


def _taken(dtype, k, rows, cols, c=1000):
    """Filters of one atom; at most four sets of rows; columns of one MMA and of the accumulators.  (Filter rows that fit one
    reduction block with their c channels are folded: one column.)"""
    atom = 64 if dtype == np.float16 else 32
    unit = 8 if dtype == np.float16 else 4
    if cols > 1 and max(cols, 2) * (-(-c // unit) * unit) <= atom:
        cols = 1
    sets = -(-rows // (128 // atom))
    return k <= atom and rows > 1 and sets <= 4 and cols * atom <= 256 and sets * cols * atom <= 512


def _run(dtype, xs, k, ks, s=1, d=1, g=1, pad="half", splits=0, flip=True, want_rows=True):
    """Values -1, 0, 1: sums below 2048 are whole numbers in both types, so nothing has to be tolerated."""
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    ctx.set_splits(splits)
    rs = np.random.RandomState(xs[1] + k + ks[0])
    kw = dict(border_mode=pad, subsample=(s, s), filter_dilation=(d, d), num_groups=g, filter_flip=flip)
    x = rs.randint(-1, 2, xs).astype(dtype)
    ho, wo = O.conv2d(np.zeros((1, g) + xs[2:], np.float32), np.zeros((g, 1) + ks, np.float32), **kw).shape[2:]
    dy = rs.randint(-1, 2, (xs[0], k, ho, wo)).astype(dtype)
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), ks, **kw)
    assert np.abs(want).max() < 2048
    got = shim.device_grad_weights(X, DY, ks, flags=shim.ROWS, **kw).to_host()
    assert (ctx.last_variant == "wgrad rows") == want_rows, ctx.last_variant
    assert np.array_equal(got, want.astype(dtype))
    ctx.close()


@DTYPES
@pytest.mark.parametrize("c,k", [(8, 4), (24, 31), (32, 32), (40, 20), (100, 7)])
@pytest.mark.parametrize("ks,h,w", [((3, 3), 14, 14), ((2, 3), 5, 41), ((5, 4), 20, 9), ((7, 1), 9, 33), ((4, 2), 3, 3), ((3, 1), 60, 58)])
def test_filter_shapes(dtype, c, k, ks, h, w):
    _run(dtype, (3, c, h, w), k, ks, pad="full" if min(h, w) < 4 else "half", want_rows=_taken(dtype, k, *ks, c=c))


@pytest.mark.parametrize("c,k", [(64, 64), (33, 50), (130, 40)])
@pytest.mark.parametrize("ks,h,w", [((3, 3), 56, 56), ((3, 3), 7, 7), ((8, 2), 16, 20), ((2, 4), 10, 11)])
def test_float16_atoms(c, k, ks, h, w):
    _run(np.float16, (2, c, h, w), k, ks, splits=3)


@DTYPES
@pytest.mark.parametrize("s,d,pad", [(2, 1, "half"), (1, 2, "half"), (2, 2, "valid"), (2, 1, ((1, 2), (2, 1))), (3, 1, "full"), (1, 3, "full")])
def test_strides_dilations_borders(dtype, s, d, pad):
    _run(dtype, (5, 16, 23, 19), 24, (3, 3), s=s, d=d, pad=pad, flip=False, want_rows=s < 3)


@DTYPES
@pytest.mark.parametrize("c,k,g", [(64, 64, 8), (256, 256, 32), (48, 24, 6), (96, 32, 2), (32, 64, 4), (64, 128, 2)])
@pytest.mark.parametrize("s", [1, 2])
def test_merged_groups(dtype, c, k, g, s):
    _run(dtype, (3, c, 12, 17), k, (3, 3), s=s, g=g, want_rows=_taken(dtype, k // g, 4 - s, 4 - s))


@DTYPES
@pytest.mark.parametrize("k", [9, 32, 60])
@pytest.mark.parametrize("ks,s,h,w", [((3, 3), 1, 30, 31), ((5, 2), 2, 17, 40), ((4, 3), 3, 25, 25)])
def test_folded_rows(dtype, k, ks, s, h, w):
    _run(dtype, (4, 3, h, w), k, ks, s=s, want_rows=_taken(dtype, k, ks[0] - (s > 1), 1))


@pytest.mark.parametrize("k,want", [(64, True), (20, True), (65, False)])
def test_pixel_blocks_of_the_stem(k, want):
    _run(np.float16, (2, 3, 46, 52), k, (7, 7), s=2, pad=(3, 3), want_rows=want)


@DTYPES
@pytest.mark.parametrize("xs,k,ks", [((2, 16, 9, 9), 65, (3, 3)), ((2, 16, 9, 9), 16, (1, 3)), ((1, 8, 3, 300), 8, (3, 3))])
def test_layers_it_does_not_take(dtype, xs, k, ks):
    _run(dtype, xs, k, ks, want_rows=False)


@DTYPES
def test_it_may_be_the_timed_choice(dtype):
    """Timed: the three kernels agree with the oracle whichever wins, and the choice is kept."""
    ctx = shim.Context(0)
    rs = np.random.RandomState(3)
    x, dy = (rs.randint(-1, 2, (2, 32, 28, 28)).astype(dtype) for _ in range(2))
    X, DY = (shim.DeviceTensor.from_host(ctx, a, "nhwc") for a in (x, dy))
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), (3, 3), border_mode="half")
    kernels = []
    for _ in range(2):
        assert np.array_equal(shim.device_grad_weights(X, DY, (3, 3), border_mode="half").to_host(), want.astype(dtype))
        kernels.append(ctx.last_variant)
    assert kernels[0] == kernels[1] and kernels[0].startswith("wgrad ")
    ctx.close()
