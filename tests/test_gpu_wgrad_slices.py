"""Slice counts that gradWeights calls remember: one layer in several forms on one context, and counts out of a file.  A count
with more slices than the pixel tiles fill would add up accumulators that nothing was written to."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


def _layer(ctx, dtype, xs, k, ks, **kw):
    """Device operands of values -1, 0, 1 and the exact gradient (whole numbers below 2048 in both types)."""
    rs = np.random.RandomState(xs[2] + k)
    x = rs.randint(-1, 2, xs).astype(dtype)
    ho, wo = O.conv2d(np.zeros((1, 1) + xs[2:], np.float32), np.zeros((1, 1) + ks, np.float32), **kw).shape[2:]
    dy = (rs.randint(-1, 2, (xs[0], k, ho, wo)) * (rs.random_sample((xs[0], k, ho, wo)) < 0.25)).astype(dtype)
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), ks, **kw)
    assert np.abs(want).max() < 2048
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")
    return (lambda flags=0: shim.device_grad_weights(X, DY, ks, flags=flags, **kw).to_host()), want.astype(dtype)


@DTYPES
@pytest.mark.parametrize("order", [(0, shim.NO_S2D), (shim.NO_S2D, 0)], ids=["blocks-first", "blocks-last"])
@pytest.mark.parametrize("n,h,k,ks", [(8, 64, 32, 4), (8, 128, 32, 4), (16, 64, 20, 4), (8, 46, 30, 3), (2, 64, 32, 5)])
def test_forms_of_one_layer(dtype, order, n, h, k, ks):
    """Pixel blocks and folded rows of a stride-2 layer cut an image into different numbers of tiles."""
    ctx = shim.Context(0)
    run, want = _layer(ctx, dtype, (n, 3, h, h), k, (ks, ks), border_mode=(1, 1), subsample=(2, 2))
    for flags in order + order:
        assert np.array_equal(run(flags), want)
    ctx.close()


@DTYPES
@pytest.mark.parametrize("factor", [1, 3, 1000])
@pytest.mark.parametrize("xs,k,ks,flags", [((8, 3, 64, 64), 32, (4, 4), shim.ROWS), ((3, 40, 20, 9), 24, (3, 3), shim.ROWS), ((3, 40, 20, 9), 24, (3, 3), 0),
                                           ((3, 40, 20, 9), 24, (3, 3), shim.NO_GROUP), ((2, 260, 9, 9), 300, (2, 2), shim.NO_GROUP)])
def test_counts_out_of_a_file(tmp_path, dtype, factor, xs, k, ks, flags):
    path, kw = str(tmp_path / "tuning"), dict(border_mode=(1, 1))
    ctx = shim.Context(0)
    run, want = _layer(ctx, dtype, xs, k, ks, **kw)
    assert np.array_equal(run(flags), want)
    ctx.tuning_save(path)
    ctx.close()
    lines = [l.split() for l in open(path).read().splitlines()]
    assert any(l[0] == "s" for l in lines)
    with open(path, "w") as f:
        f.writelines(" ".join(l[:2] + [str(int(l[2]) * factor)] if l[0] == "s" else l) + "\n" for l in lines)
    ctx = shim.Context(0)
    ctx.tuning_load(path)
    run, want = _layer(ctx, dtype, xs, k, ks, **kw)
    assert np.array_equal(run(flags), want)
    ctx.close()
