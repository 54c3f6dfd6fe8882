"""Filter packing in 16-byte pieces: banks off the 16-byte boundaries, runs of every alignment, block-diagonal banks of
merged groups packed from the layer's own filters, and patches cut small because the bank is."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])


def check(dtype, c, k, g, kernel, stride=1, shift=0):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(c * 31 + k + g + shift)
    x = rs.standard_normal((2, c, 12, 10)).astype(dtype)
    w = (rs.standard_normal((k, c // g) + kernel) / np.sqrt(c // g * kernel[0] * kernel[1])).astype(dtype)
    kw = dict(border_mode="half", subsample=(stride, stride), num_groups=g)
    es = w.itemsize
    X = shim.DeviceTensor.from_host(ctx, x, "nhwc")
    block = shim.DeviceTensor(ctx, (1, 1, 1, w.size + 16 // es), dtype)
    W = shim.DeviceTensor(ctx, w.shape, dtype, _ptr=block.ptr + shift * es)
    ctx.h2d(W.ptr, w)
    y = shim.device_conv2d(X, W, **kw)
    dy = rs.standard_normal(y.shape).astype(dtype)
    dx = shim.device_grad_inputs(W, shim.DeviceTensor.from_host(ctx, dy, "nhwc"), x.shape[2:], **kw).to_host()
    f = np.float32
    # the repository's bounds: 5e-3 of the largest result with TF32 factors, 2e-2 with float16 tensors
    tol = 5e-3 if dtype == np.float32 else 2e-2
    assert O.rel_err(y.to_host().astype(f), O.conv2d(x.astype(f), w.astype(f), **kw)) < tol
    assert O.rel_err(dx.astype(f), O.conv2d_grad_inputs(w.astype(f), dy.astype(f), x.shape[2:], **kw)) < tol


@DTYPES
@pytest.mark.parametrize("shift", [1, 3])
@pytest.mark.parametrize("c,k,kernel", [(16, 16, (3, 3)), (40, 33, (1, 1)), (21, 70, (5, 3)), (8, 64, (8, 8))])
def test_banks_off_the_16_byte_boundaries(dtype, c, k, kernel, shift):
    check(dtype, c, k, 1, kernel, shift=shift)


@DTYPES
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("c,k,g,kernel,stride", [(64, 64, 8, (3, 3), 1), (48, 96, 6, (1, 1), 1), (128, 32, 4, (5, 5), 2), (72, 216, 9, (2, 3), 1),
                                                 (4, 8, 2, (3, 3), 1), (8, 16, 4, (3, 3), 2)])
def test_merged_groups_are_packed_from_their_own_filters(dtype, c, k, g, kernel, stride, shift):
    check(dtype, c, k, g, kernel, stride, shift)


@DTYPES
@pytest.mark.parametrize("c,k", [(1, 1), (8, 8), (31, 9), (130, 257), (512, 300)])
@pytest.mark.parametrize("kernel", [(1, 1), (3, 3)])
def test_patches_of_small_and_large_banks(dtype, c, k, kernel):
    check(dtype, c, k, 1, kernel)
