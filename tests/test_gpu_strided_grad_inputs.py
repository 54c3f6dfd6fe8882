"""gradInputs of strided layers: all parity classes of dx in one launch against class by class and the oracle."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor
TOL = {np.float32: 5e-3, np.float16: 2e-2}      # the repository's bounds: TF32 factors, float16 tensors

# (input, filters, taps, strides, dilation): classes of one to four taps and of unequal extents (odd sizes), two and four
# classes, channels of one and more tiles, odd filter counts; the last ones have an empty class or too many classes
LAYERS = [((6, 64, 28, 28), 128, (3, 3), (2, 2), 1), ((5, 64, 27, 31), 33, (3, 3), (2, 2), 1), ((3, 192, 15, 14), 96, (3, 3), (2, 2), 1),
          ((4, 128, 20, 21), 64, (5, 4), (2, 2), 1), ((4, 64, 19, 18), 40, (3, 3), (2, 1), 1), ((4, 64, 18, 19), 40, (2, 3), (1, 2), 1),
          ((2, 320, 13, 13), 64, (2, 2), (2, 2), 1), ((70, 64, 9, 9), 64, (3, 3), (2, 2), 1), ((3, 64, 30, 30), 64, (7, 7), (2, 2), 1),
          ((3, 64, 21, 21), 64, (4, 4), (3, 1), 1), ((3, 64, 21, 21), 64, (1, 1), (2, 2), 1), ((3, 64, 21, 21), 64, (3, 3), (2, 2), 2),
          ((3, 64, 21, 21), 64, (5, 5), (3, 2), 1), ((3, 40, 21, 21), 64, (3, 3), (2, 2), 1)]


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("xs,k,ks,s,d", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_classes_together_equal_class_by_class_and_the_oracle(dtype, xs, k, ks, s, d):
    rs = np.random.RandomState(k)
    f = np.float32
    kw = dict(border_mode="half", subsample=s, filter_dilation=(d, d))
    w = (rs.standard_normal((k, xs[1]) + ks) / np.sqrt(k * ks[0] * ks[1])).astype(dtype)
    yshape = shim.hostlogic.forward_shape(xs, w.shape, "half", s, (d, d), 1)[0]
    dy = rs.standard_normal(yshape).astype(dtype)
    want = O.conv2d_grad_inputs(w.astype(f), dy.astype(f), xs[2:], **kw)
    ctx = shim.Context(0)
    W, DY = T.from_host(ctx, w), T.from_host(ctx, dy, "nhwc")
    got = {}
    for tuned in (False, True):
        for pair in (True, False):
            for flags in (0, shim.NO_MERGE_PARITY):
                ctx.set_autotune(tuned)
                ctx.set_pair_kernels(pair)
                dx = T(ctx, xs, dtype, "nhwc")
                ctx.memset(dx.ptr, 0x7B, dx.nbytes)           # whatever is not written shows
                shim.device_grad_inputs(W, DY, xs[2:], out=dx, flags=flags, **kw)
                got[tuned, pair, flags] = dx.to_host().astype(f)
                assert O.rel_err(got[tuned, pair, flags], want) < TOL[dtype], (tuned, pair, flags)
    # the same products; a class alone may be cut into slices that are added in another order
    assert O.rel_err(got[False, True, 0], got[False, False, shim.NO_MERGE_PARITY]) < TOL[dtype] / 4
    ctx.close()
