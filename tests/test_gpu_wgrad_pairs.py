"""gradWeights on pairs of CTAs, 256 filters x 256 channels: edges of the tiles, partial last tiles, groups, stages of
every number of steps."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("c,k,g", [(256, 256, 1), (260, 264, 1), (520, 300, 1), (512, 1024, 2)])
@pytest.mark.parametrize("n,h,w,ks,s", [(3, 7, 7, 3, 1), (2, 14, 14, 3, 2), (5, 8, 8, 1, 1), (1, 3, 61, 2, 1), (1, 1, 1, 1, 1)])
def test_pairs_of_wide_layers(dtype, c, k, g, n, h, w, ks, s):
    """Values -1, 0, 1: sums below 2048 are whole numbers in both types, so nothing has to be tolerated."""
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    rs = np.random.RandomState(c + k + h)
    x = rs.randint(-1, 2, (n, c, h, w)).astype(dtype)
    kw = dict(border_mode="half", subsample=(s, s), num_groups=g)
    ho, wo = O.conv2d(x[:1, :g].astype(np.float32), np.zeros((g, 1, ks, ks), np.float32), **kw).shape[2:]
    dy = rs.randint(-1, 2, (n, k, ho, wo)).astype(dtype)
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), (ks, ks), **kw)
    dw = shim.device_grad_weights(X, DY, (ks, ks), flags=shim.NO_GROUP, **kw).to_host()
    assert np.array_equal(dw, want.astype(dtype))
    ctx.close()
