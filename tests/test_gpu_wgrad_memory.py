"""gradWeights with little memory left: the kernel that stacks filter rows wants a slab for each of its many slices, the others
fewer; where its slabs do not fit, the call runs without it."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor
MB = 1 << 20
LAYERS = {"plain": (np.float32, (64, 32, 28, 28), 32, 5, 1), "groups": (np.float32, (64, 32, 28, 28), 32, 5, 2),
          "folded": (np.float16, (127, 1, 28, 28), 64, 7, 1)}      # 99568 output pixels: timed


@pytest.mark.parametrize("tuned", [False, True], ids=["untimed", "timed"])
@pytest.mark.parametrize("form", sorted(LAYERS))
def test_without_memory_for_the_slabs_of_stacked_rows(form, tuned):
    dtype, xs, k, ks, g = LAYERS[form]
    kw = dict(border_mode="half", num_groups=g)
    rs = np.random.RandomState(1)
    x, dy = rs.randint(-1, 2, xs).astype(dtype), rs.randint(-1, 2, (xs[0], k) + xs[2:]).astype(dtype)
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), (ks, ks), **kw)      # whole numbers: exact in float32

    def context(tuned):
        c = shim.Context(0)
        c.set_autotune(tuned)
        X, DY, DW = T.from_host(c, x, "nhwc"), T.from_host(c, dy, "nhwc"), T(c, want.shape, np.float32)
        return c, DW, lambda flags=0: shim.device_grad_weights(X, DY, (ks, ks), out=DW, flags=flags, **kw)

    def scratch(tuned, flags):
        """Bytes that a call takes (and the kernels' code, which has to be on the device before its memory is taken)."""
        c, _, run = context(tuned)
        before = c.memory_info()[0]
        run(flags)
        assert (c.last_variant == "wgrad rows") == (flags == shim.ROWS)
        need = c.memory_info()[0] - before
        c.close()
        return need

    rows, others = scratch(False, shim.ROWS), max(scratch(tuned, f) for f in (shim.NO_ROWS, shim.NO_GROUP))
    spare = others + 2 * MB
    assert rows > spare + 4 * MB, (rows, others)
    c, DW, run = context(tuned)
    block, taken, size = T(c, (1, 1, 1, spare // 4), np.float32), [], 256 << 30
    while size >= 2 * MB:
        try:
            taken.append(T(c, (1, 1, 1, size // 4), np.float32))
        except (MemoryError, shim.B200Error):
            size //= 2
    try:
        assert c.memory_info()[1] < 4 * MB
        block.free()
        for flags in (0, shim.ROWS):
            run(flags)
            assert c.last_variant != "wgrad rows"
            c.sync()
    except BaseException:
        c.close()                                           # gives the device its memory back before other tests run
        raise
    for t in taken:
        t.free()
    assert np.array_equal(DW.to_host(), want)
    run(shim.ROWS)
    assert c.last_variant == "wgrad rows" and np.array_equal(DW.to_host(), want)
    before = c.launches
    run()
    if tuned:
        assert c.launches - before > 5                      # what was chosen for want of memory is not remembered
    assert np.array_equal(DW.to_host(), want)
    c.close()
