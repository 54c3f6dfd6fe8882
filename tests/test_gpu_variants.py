"""Which kernel variant runs: the geometries of the pair and class tests are meant to take pairs of CTAs and one launch for
all classes, and a change of the models must not leave those tests comparing a kernel with itself."""
import numpy as np
import pytest

import test_gpu_slab_pairs as pairs
import test_gpu_strided_grad_inputs as strided
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


@pytest.fixture
def ctx():
    c = shim.Context(0)
    c.set_autotune(False)
    yield c
    c.close()


@DTYPES
@pytest.mark.parametrize("xs,k,ks,g,d", pairs.LAYERS[1:], ids=lambda v: str(v).replace(" ", ""))     # the first has few tiles
def test_pair_layers_run_on_pairs(ctx, dtype, xs, k, ks, g, d):
    X, W = T(ctx, xs, dtype, "nhwc"), T(ctx, (k, xs[1] // g, ks, ks), dtype)
    kw = dict(border_mode="half", num_groups=g, filter_dilation=(d, d))
    for layout in ("nhwc", "nchw"):
        shim.device_conv2d(X, W, out_layout=layout, **kw)
        assert ctx.last_variant == "slab pair"
    ctx.set_pair_kernels(False)
    shim.device_conv2d(X, W, **kw)
    assert ctx.last_variant == "slab"


@DTYPES
@pytest.mark.parametrize("n", [16, 17])
def test_pooling_layers_run_on_pairs(ctx, dtype, n):
    X, W = T(ctx, (n, 48, 36, 36), dtype, "nhwc"), T(ctx, (128, 48, 3, 3), dtype)
    shim.device_conv2d(X, W, border_mode="half", relu=True, pool=True)
    assert ctx.last_variant == "slab pair"


@DTYPES
@pytest.mark.parametrize("xs,k,ks,s,d", strided.LAYERS, ids=lambda v: str(v).replace(" ", ""))
def test_strided_grad_inputs_take_one_launch_for_all_classes(ctx, dtype, xs, k, ks, s, d):
    """Where every class has a tap, there are at most four and the channels are whole 128-byte chunks."""
    taps = [{(-i * d + (ks[a] - 1) * d // 2) % s[a] for i in range(ks[a])} for a in range(2)]
    whole = all(len(taps[a]) == s[a] for a in range(2)) and s[0] * s[1] <= 4 and xs[1] * np.dtype(dtype).itemsize % 128 == 0
    yshape = shim.hostlogic.forward_shape(xs, (k, xs[1]) + ks, "half", s, (d, d), 1)[0]
    W, DY = T(ctx, (k, xs[1]) + ks, dtype), T(ctx, yshape, dtype, "nhwc")
    for pair in (True, False):
        ctx.set_pair_kernels(pair)
        shim.device_grad_inputs(W, DY, xs[2:], border_mode="half", subsample=s, filter_dilation=(d, d))
        assert ctx.last_variant.startswith("slab classes") == whole and (pair or "pair" not in ctx.last_variant)
        shim.device_grad_inputs(W, DY, xs[2:], border_mode="half", subsample=s, filter_dilation=(d, d), flags=shim.NO_MERGE_PARITY)
        assert "classes" not in ctx.last_variant


@DTYPES
def test_split_layers_run_split(ctx, dtype):
    X, W = T(ctx, (1, 512, 14, 14), dtype, "nhwc"), T(ctx, (512, 512, 3, 3), dtype)
    for flags, variant in ((0, "slab split"), (shim.NO_SLAB, "tap split")):
        shim.device_conv2d(X, W, border_mode="half", flags=flags)
        assert ctx.last_variant == variant


def test_choices_of_a_file_hold_for_the_switch_they_were_made_with(tmp_path):
    """A file that names pairs for a geometry does not bring them to a context that has them switched off."""
    path = str(tmp_path / "tuning")
    xs, ws = (40, 512, 14, 14), (512, 512, 3, 3)
    for step in ("make", "on", "off"):
        c = shim.Context(0)
        X, W = T(c, xs, np.float32, "nhwc"), T(c, ws, np.float32)
        if step != "make":
            c.set_pair_kernels(step == "on")
            assert c.tuning_load(path) == 1
        shim.device_conv2d(X, W, border_mode="half")
        if step == "make":
            c.tuning_save(path)
            head, line = open(path).read().splitlines()
            open(path, "w").write("\n".join([head, " ".join(line.split()[:2] + ["4"])]) + "\n")      # pairs, whatever was faster
        else:
            shim.device_conv2d(X, W, border_mode="half")
            assert (c.last_variant == "slab pair") == (step == "on")
        c.close()
