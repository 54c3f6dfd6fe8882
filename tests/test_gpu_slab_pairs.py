"""The slab kernel on pairs of CTAs: two pixel tiles side by side, each CTA with half of the filter tile."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor
TOL = {np.float32: 5e-3, np.float16: 2e-2}      # the repository's bounds: TF32 factors, float16 tensors

# (images, filters, taps per side, groups, dilation): filters at the edges of 64, 128 and 256 columns, tile counts odd and
# even (the last pair's second tile then lies behind the last image), tap counts that leave a remainder in a stage
LAYERS = [((5, 64, 30, 30), 64, 3, 1, 1), ((37, 100, 27, 33), 75, 5, 1, 1), ((9, 96, 28, 28), 256, 3, 1, 1), ((3, 256, 56, 56), 130, 3, 1, 1),
          ((40, 512, 14, 14), 512, 3, 1, 1), ((12, 40, 41, 40), 200, 2, 1, 1), ((33, 64, 17, 19), 320, 1, 1, 1), ((64, 64, 28, 28), 128, 3, 2, 1),
          ((7, 33, 50, 21), 300, 3, 1, 2), ((151, 256, 7, 7), 129, 3, 1, 1)]


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("xs,k,ks,g,d", LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_pairs_equal_single_ctas_and_the_oracle(dtype, xs, k, ks, g, d):
    rs = np.random.RandomState(k)
    f = np.float32
    x = rs.standard_normal(xs).astype(dtype)
    w = (rs.standard_normal((k, xs[1] // g, ks, ks)) / np.sqrt(xs[1] // g * ks * ks)).astype(dtype)
    b = rs.standard_normal(k).astype(dtype)
    kw = dict(border_mode="half", num_groups=g, filter_dilation=(d, d))
    want_y = O.bias_relu(O.conv2d(x.astype(f), w.astype(f), **kw), b.astype(f), relu=True)
    want_dx = None
    got = {}
    ctx = shim.Context(0)
    ctx.set_autotune(False)                     # the model's choice: pairs, where they are allowed and occupy half of the SMs
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b.reshape(1, k, 1, 1))
    for pair in (True, False):
        ctx.set_pair_kernels(pair)
        for layout in ("nhwc", "nchw"):
            Y = shim.device_conv2d(X, W, bias=B, relu=True, out_layout=layout, **kw)
            got[pair, layout] = Y.to_host().astype(f)
            assert O.rel_err(got[pair, layout], want_y) < TOL[dtype], (pair, layout)
            if layout == "nhwc":
                DX = shim.device_grad_inputs(W, Y, xs[2:], **kw)
                if want_dx is None:
                    want_dx = O.conv2d_grad_inputs(w.astype(f), Y.to_host().astype(f), xs[2:], **kw)
                got[pair, "dx"] = DX.to_host().astype(f)
                assert O.rel_err(got[pair, "dx"], want_dx) < TOL[dtype], pair
    # the same products; only a tile whose reduction is cut elsewhere adds them in another order
    for what in ("nhwc", "nchw", "dx"):
        assert O.rel_err(got[True, what], got[False, what]) < TOL[dtype] / 4, what
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("n", [16, 17])
def test_pairs_pool_in_the_epilogue(dtype, n):
    rs = np.random.RandomState(n)
    f = np.float32
    x = rs.standard_normal((n, 48, 36, 36)).astype(dtype)
    w = (rs.standard_normal((128, 48, 3, 3)) / 20).astype(dtype)
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    X, W = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w)
    got = []
    for pair in (True, False):
        ctx.set_pair_kernels(pair)
        got.append(shim.device_conv2d(X, W, border_mode="half", relu=True, pool=True).to_host().astype(f))
    want = O.maxpool2x2(np.maximum(O.conv2d(x.astype(f), w.astype(f), border_mode="half", subsample=(1, 1)), 0))
    assert O.rel_err(got[0], want) < TOL[dtype] and O.rel_err(got[0], got[1]) < TOL[dtype] / 4
    ctx.close()


def test_switching_pairs_off_holds_for_geometries_timed_before(tmp_path):
    ctx = shim.Context(0)
    X = T.from_host(ctx, np.ones((40, 512, 14, 14), np.float32), "nhwc")
    W = T.from_host(ctx, np.ones((512, 512, 3, 3), np.float32))

    def choices():
        shim.device_conv2d(X, W, border_mode="half")
        ctx.tuning_save(str(tmp_path / "t"))
        return [l.split() for l in open(str(tmp_path / "t")) if l.startswith("a ")]
    on = choices()
    ctx.set_pair_kernels(False)
    off = [c for c in choices() if c not in on]
    assert len(on) == 1 and len(off) == 1 and off[0][2] != "4"           # a choice of its own, and not the pairs
    ctx.close()
