"""The first call of a geometry times the kernel variants; how many launches that may take."""
import numpy as np
import pytest

from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
def test_first_calls_do_not_time_what_is_far_behind(dtype):
    """Strided gradInputs: three forms, one of which is a launch for each of four classes with choices of its own.
    Eighteen runs of everything took 340 launches and more.  Now: the packing, two runs of each form (2 x 4, 2, 2), two
    of each of the two together (2 x 2), two bursts of at most 8 of each where they are close (2 x 16), the result: 49."""
    ctx = shim.Context(0)
    rs = np.random.RandomState(0)
    n, c, k, h = 32, 64, 64, 56
    W = T.from_host(ctx, rs.standard_normal((k, c, 3, 3)).astype(dtype))
    DY = T.from_host(ctx, rs.standard_normal((n, k, h // 2, h // 2)).astype(dtype), "nhwc")
    before = ctx.launches
    first = shim.device_grad_inputs(W, DY, (h, h), border_mode="half", subsample=(2, 2)).to_host()
    tuning = ctx.launches - before
    before = ctx.launches
    again = shim.device_grad_inputs(W, DY, (h, h), border_mode="half", subsample=(2, 2))
    assert ctx.launches - before <= 2 and tuning <= 49, tuning
    assert np.array_equal(first, again.to_host())
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("n,c,k,h,ks", [(8, 64, 64, 28, 3), (128, 256, 256, 14, 3), (37, 100, 75, 29, 5), (4, 32, 32, 56, 3), (1, 512, 512, 28, 3)])
def test_first_forward_calls_run_every_variant_twice_and_few_in_bursts(dtype, n, c, k, h, ks):
    """Stride 1: up to eight variants.  The packing, two runs of each (two launches where the reduction is split), two bursts of at most 7 of those
    within a fifth of the best, the result.  Measured 18 to 71; all eight in both bursts would be 130 and more."""
    ctx = shim.Context(0)
    rs = np.random.RandomState(0)
    X = T.from_host(ctx, rs.standard_normal((n, c, h, h)).astype(dtype), "nhwc")
    W = T.from_host(ctx, (rs.standard_normal((k, c, ks, ks)) / np.sqrt(c * ks * ks)).astype(dtype))
    before = ctx.launches
    first = shim.device_conv2d(X, W, border_mode="half").to_host()
    tuning = ctx.launches - before
    before = ctx.launches
    again = shim.device_conv2d(X, W, border_mode="half")
    assert ctx.launches - before <= 3 and tuning <= 90, tuning
    assert np.array_equal(first, again.to_host())
    ctx.close()
