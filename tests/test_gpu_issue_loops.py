"""The issue loops of the tensor-core kernels: every number of taps per stage with straight-line code and the loops for the
others, one and two accumulators per issuing warp, stages of every number of reduction steps."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


@pytest.fixture(scope="module")
def ctx():
    c = shim.Context(0)
    c.set_autotune(False)
    yield c
    c.close()


def _ints(rs, shape, dtype):
    """Values -1, 0, 1: products and sums below 2048 are whole numbers that every type here holds, so that the result is
    the same in any order of accumulation and nothing has to be tolerated."""
    return rs.randint(-1, 2, shape).astype(dtype)


@DTYPES
@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("k", [20, 64, 96, 160])                  # tiles of 32, 64, 128 and 256 filters
@pytest.mark.parametrize("ks", [(1, 1), (1, 2), (1, 3), (2, 2), (1, 5), (7, 1), (3, 3), (3, 5), (5, 5)])
def test_taps_per_stage(ctx, dtype, pairs, k, ks):
    ctx.set_pair_kernels(pairs)
    rs = np.random.RandomState(k + ks[0] * 10 + ks[1])
    x = _ints(rs, (9, 70, 19, 23), dtype)                         # channels: three float32 blocks, two float16 blocks
    w = _ints(rs, (k, 70) + ks, dtype)
    X, W = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, w)
    y = shim.device_conv2d(X, W, border_mode="half").to_host()
    want = O.conv2d(x.astype(np.float32), w.astype(np.float32), border_mode="half")
    assert np.array_equal(y, want.astype(dtype))
    dx = shim.device_grad_inputs(W, shim.DeviceTensor.from_host(ctx, y, "nhwc"), (19, 23), border_mode="half")
    small = _ints(rs, y.shape, dtype)
    dx = shim.device_grad_inputs(W, shim.DeviceTensor.from_host(ctx, small, "nhwc"), (19, 23), border_mode="half", out=dx).to_host()
    want = O.conv2d_grad_inputs(w.astype(np.float32), small.astype(np.float32), (19, 23), border_mode="half")
    assert np.abs(want).max() < 2048 and np.array_equal(dx, want.astype(dtype))


@DTYPES
@pytest.mark.parametrize("c,k", [(24, 40), (64, 130), (100, 75), (260, 30)])
@pytest.mark.parametrize("h,w,ks", [(5, 6, 3), (9, 30, 2), (12, 56, 3), (3, 61, 4), (2, 130, 3), (11, 13, 1)])
def test_reduction_steps_per_stage(ctx, dtype, c, k, h, w, ks):
    """Widths that give stages of few, seven and eight steps, whole rows and segments."""
    rs = np.random.RandomState(h * w + ks)
    n = max(1, 1500 // (h * w))
    x = _ints(rs, (n, c, h, w), dtype)
    dy = _ints(rs, (n, k, h + ks - 1, w + ks - 1), dtype)         # 'full' borders
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), (ks, ks), border_mode="full")
    assert np.abs(want).max() < 2048
    for flags in (0, shim.NO_GROUP):
        dw = shim.device_grad_weights(X, DY, (ks, ks), border_mode="full", flags=flags).to_host()
        assert np.array_equal(dw, want.astype(dtype))
