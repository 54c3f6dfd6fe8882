"""gradWeights of float32 layers with at most 64 channels: the taps of a filter row as column groups of one MMA per 32
channels, against one MMA per tap (the same products in the same order) and the oracle."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

# (images, filters, taps per side, stride, dilation): channels at the edges of one and two atoms; groups of one to four taps
LAYERS = [((8, 64, 14, 14), 64, 3, 1, 1), ((5, 32, 17, 17), 96, 3, 1, 1), ((4, 33, 12, 12), 128, 5, 1, 1), ((4, 48, 16, 16), 130, 3, 1, 2),
          ((4, 64, 15, 15), 64, 3, 2, 1), ((3, 8, 30, 9), 20, 3, 1, 1), ((2, 64, 70, 70), 128, 2, 1, 1), ((2, 40, 13, 90), 7, 7, 1, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("xs,k,ks,s,d", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_stacked_taps_equal_single_taps_and_the_oracle(xs, k, ks, s, d):
    ctx = shim.Context(0)
    rs = np.random.RandomState(33)
    pad = (ks // 2) * d
    kw = dict(border_mode=(pad, pad), subsample=(s, s), filter_dilation=(d, d))
    x = rs.standard_normal(xs).astype(np.float32)
    ho, wo = ((n + 2 * pad - ((ks - 1) * d + 1)) // s + 1 for n in xs[2:])
    dy = (rs.standard_normal((xs[0], k, ho, wo)) * 0.1).astype(np.float32)
    want = O.conv2d_grad_weights(x, dy, (ks, ks), **kw)
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")
    ctx.set_autotune(False)
    got = {}
    for stacked in (True, False):
        ctx.set_stacked_taps(stacked)
        for splits in (0, 1, 3):
            ctx.set_splits(splits)
            got[stacked, splits] = shim.device_grad_weights(X, DY, (ks, ks), flags=shim.FORCE_UMMA, **kw).to_host()
            assert O.rel_err(got[stacked, splits], want) < 5e-3          # the repository's bound: TF32 factors
    for splits in (0, 1, 3):
        assert np.array_equal(got[True, splits], got[False, splits])
    ctx.close()
