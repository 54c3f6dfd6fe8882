"""The read-out of the per-tap kernel: several tiles per CTA (rows leave through transpose buffers in float32), one tile per CTA,
narrow tiles whose warps take turns, partial last tiles, residual, bias and activation."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("n,h,w", [(150, 13, 17), (2, 9, 8)])           # 260 pixel tiles, 2 of them
@pytest.mark.parametrize("k", [4, 20, 36, 64, 100, 132, 260])
@pytest.mark.parametrize("s", [1, 2])
def test_read_out(dtype, n, h, w, k, s):
    """Values -1, 0, 1: sums below 2048 are whole numbers in both types, so nothing has to be tolerated."""
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    rs = np.random.RandomState(k + h + s)
    T = shim.DeviceTensor.from_host
    x, wt = rs.randint(-1, 2, (n, 24, h, w)).astype(dtype), rs.randint(-1, 2, (k, 24, 3, 3)).astype(dtype)
    b = rs.randint(-3, 4, (k,)).astype(dtype)
    kw = dict(border_mode="half", subsample=(s, s))
    conv = O.conv2d(x.astype(np.float32), wt.astype(np.float32), **kw)
    r = rs.randint(-5, 6, conv.shape).astype(dtype)
    X, W = T(ctx, x, "nhwc"), T(ctx, wt)
    B, R = T(ctx, b.reshape(1, k, 1, 1)), T(ctx, r, "nhwc")
    got = shim.device_conv2d(X, W, flags=shim.NO_SLAB, **kw)
    assert ctx.last_variant.startswith("tap")
    assert np.array_equal(got.to_host(), conv.astype(dtype))
    got = shim.device_conv2d(X, W, bias=B, relu=True, flags=shim.NO_SLAB, **kw)
    assert np.array_equal(got.to_host(), np.maximum(conv + b.reshape(1, k, 1, 1).astype(np.float32), 0).astype(dtype))
    got = shim.device_conv2d(X, W, residual=R, beta=2.0, flags=shim.NO_SLAB, **kw)
    assert np.array_equal(got.to_host(), (conv + 2 * r.astype(np.float32)).astype(dtype))
    ctx.close()
