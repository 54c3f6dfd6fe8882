"""gradInputs of stride-2 layers with up to four channels: the classes of the stride written straight to the gradient's pixels, or by
way of a tensor of classes, where images end inside a 2x2 block, kernels are even, odd or wider than tall, and filters are few or many."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
T = shim.DeviceTensor
F = np.float32


@DTYPES
@pytest.mark.parametrize("c", [1, 3, 4])
@pytest.mark.parametrize("n,h,w_,k,ks", [(2, 31, 45, 64, (7, 7)), (3, 16, 66, 20, (4, 4)), (1, 130, 33, 70, (3, 5)), (40, 24, 25, 33, (2, 3)),
                                         (2, 20, 20, 8, (8, 8)), (2, 9, 9, 300, (3, 3)), (150, 18, 17, 16, (5, 5))])
def test_against_the_oracle(dtype, c, n, h, w_, k, ks):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(n + k + c)
    kw = dict(border_mode="half", subsample=(2, 2))
    w = (rs.standard_normal((k, c) + ks) / np.sqrt(k * ks[0] * ks[1] / 4)).astype(dtype)
    ys = shim.hostlogic.forward_shape((n, c, h, w_), w.shape, "half", (2, 2), (1, 1), 1)[0]
    dy = rs.standard_normal(ys).astype(dtype)
    W, DY = T.from_host(ctx, w), T.from_host(ctx, dy, "nhwc")
    DX = T(ctx, (n, c, h, w_), dtype, "nhwc")
    ctx.memset(DX.ptr, 255, DX.nbytes)
    shim.device_grad_inputs(W, DY, (h, w_), out=DX, **kw)
    ref = O.conv2d_grad_inputs(w.astype(F), dy.astype(F), (h, w_), **kw)
    tol = 5e-3 if dtype == F else 2e-2             # the repository's bounds for TF32 factors and float16 tensors
    assert O.rel_err(DX.to_host().astype(F), ref) < tol
    stored = np.empty((n, h, w_, ctx.padded_channels(c, dtype)), dtype)
    ctx.d2h(stored, DX.ptr)
    ctx.sync()
    assert not stored[..., c:].any()               # pad channels
