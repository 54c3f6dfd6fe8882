"""MMAs as wide as a tile has filters: counts around the steps of 16 (single CTAs) and 32 (pairs) columns, alone in a tile and in the
last of several, on the slab kernel, its pairs, split reductions and the per-tap kernel."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
T = shim.DeviceTensor


@DTYPES
@pytest.mark.parametrize("k", [33, 48, 65, 80, 97, 112, 130, 160, 257, 273, 300])
@pytest.mark.parametrize("n", [1, 14])
def test_filter_counts_off_the_tile_widths(dtype, n, k):
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    rs = np.random.RandomState(k + n)
    x = rs.standard_normal((n, 24, 28, 28)).astype(dtype)
    w = (rs.standard_normal((k, 24, 3, 3)) / np.sqrt(24 * 9)).astype(dtype)
    b = rs.standard_normal((1, k, 1, 1)).astype(dtype)
    f = np.float32
    ref = np.maximum(O.conv2d(x.astype(f), w.astype(f), border_mode="half") + b.astype(f), 0)
    X, W, B = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T.from_host(ctx, b)
    seen = set()
    for pair, flags, layout in ((True, 0, "nhwc"), (False, 0, "nhwc"), (False, 0, "nchw"), (True, shim.NO_SLAB, "nhwc")):
        ctx.set_pair_kernels(pair)
        y = shim.device_conv2d(X, W, border_mode="half", bias=B, relu=True, out_layout=layout, flags=flags).to_host()
        seen.add(ctx.last_variant)
        # the repository's bounds: 5e-3 of the largest result with TF32 factors, 2e-2 with float16 tensors
        assert O.rel_err(y.astype(f), ref) < (5e-3 if dtype == np.float32 else 2e-2), ctx.last_variant
    assert any(v.startswith("tap") for v in seen) and any(v.startswith("slab") for v in seen)
    assert n == 1 or "slab pair" in seen
    ctx.close()


# channels whose filter rows are whole 128-byte blocks (narrow MMAs on pairs) and others, with and without staged stores; shallow and deep
@DTYPES
@pytest.mark.parametrize("c,k,kernel", [(128, 75, 3), (64, 178, 3), (24, 75, 3), (24, 75, 5), (40, 96, 3), (24, 192, 3), (136, 192, 3), (72, 320, 3), (200, 330, 1)])
def test_pairs_with_whole_and_narrow_tiles(tmp_path, dtype, c, k, kernel):
    rs = np.random.RandomState(c + k)
    f = np.float32
    x = rs.standard_normal((14, c, 28, 28)).astype(dtype)
    w = (rs.standard_normal((k, c, kernel, kernel)) / np.sqrt(c * kernel * kernel)).astype(dtype)
    ref = O.conv2d(x.astype(f), w.astype(f), border_mode="half")
    path = str(tmp_path / "t")
    first = shim.Context(0)
    shim.device_conv2d(T.from_host(first, x, "nhwc"), T.from_host(first, w), border_mode="half")
    first.tuning_save(path)
    first.close()
    head, *rest = open(path).read().splitlines()
    for choice in (4, 5):                                # the slab and the per-tap kernel on pairs, where they take the layer
        open(path, "w").write("\n".join([head] + [" ".join(r.split()[:2] + [str(choice)]) for r in rest if r.startswith("a 3.")]) + "\n")
        ctx = shim.Context(0)
        assert ctx.tuning_load(path) == 1
        y = shim.device_conv2d(T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), border_mode="half")
        assert choice == 5 or "pair" in ctx.last_variant
        assert O.rel_err(y.to_host().astype(f), ref) < (5e-3 if dtype == f else 2e-2), ctx.last_variant
        ctx.close()
