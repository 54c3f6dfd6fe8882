"""Cut tiles whose slices are added by the CTA that leaves the last one: results repeat bit by bit over calls, graphs and contexts, and the
counts of arrivals are back at zero after a wait that ran out."""
import ctypes

import numpy as np
import pytest

from theano_b200 import shim

pytestmark = pytest.mark.gpu
T = shim.DeviceTensor


def layer(ctx, dtype):
    c = 256 if dtype == np.float32 else 512
    rs = np.random.RandomState(11)
    x = rs.standard_normal((100, c, 14, 14)).astype(dtype)
    w = (rs.standard_normal((256, c, 3, 3)) / np.sqrt(c * 9)).astype(dtype)
    X, W, Y = T.from_host(ctx, x, "nhwc"), T.from_host(ctx, w), T(ctx, (100, 256, 14, 14), dtype, "nhwc")
    return X, W, Y, lambda: shim.device_conv2d(X, W, border_mode="half", out=Y, flags=shim.NO_SLAB)


@pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
def test_repeated_calls_graphs_and_contexts_agree(dtype):
    first = None
    for _ in range(2):
        ctx = shim.Context(0)
        ctx.set_autotune(False)
        X, W, Y, call = layer(ctx, dtype)
        call()
        assert ctx.last_variant == "tap pair cut"
        y = Y.to_host()
        first = y if first is None else first
        assert np.array_equal(first, y)
        graph = ctx.capture(lambda: [call() for _ in range(5)])
        for _ in range(4):
            ctx.memset(Y.ptr, 255, Y.nbytes)
            graph.launch()
        ctx.sync()
        assert np.array_equal(first, Y.to_host())
        graph.destroy()
        ctx.close()


def test_counts_start_again_after_a_wait_ran_out():
    """The self-test leaves counts with which no cut tile would ever be complete, that is, stored."""
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    X, W, Y, call = layer(ctx, np.float32)
    call()
    y = Y.to_host()
    ctx.set_wait_limit(2000000)                      # about a millisecond
    with pytest.raises(shim.B200Error):
        ctx.selftest_wait()
    ctx.set_wait_limit(4000000000)
    for _ in range(2):
        ctx.memset(Y.ptr, 255, Y.nbytes)
        call()
        assert ctx.last_variant == "tap pair cut" and np.array_equal(y, Y.to_host())
    ctx.close()


def test_a_context_made_while_the_default_stream_is_busy():
    """The counts of a new context are zero before its first launch, whatever another library has queued on the default stream and
    whatever their memory held before."""
    torch = pytest.importorskip("torch")
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    X, W, Y, call = layer(ctx, np.float32)
    call()
    y = Y.to_host()
    cudart = ctypes.CDLL("libcudart.so.12")
    big = torch.empty(1 << 30, dtype=torch.float32, device="cuda")
    blocks = [ctypes.c_void_p() for _ in range(512)]
    for b in blocks:
        assert cudart.cudaMalloc(ctypes.byref(b), ctypes.c_size_t(4096)) == 0
        assert cudart.cudaMemset(b, 255, ctypes.c_size_t(4096)) == 0
    torch.cuda.synchronize()
    for b in blocks:
        assert cudart.cudaFree(b) == 0
    for _ in range(300):                             # some 180 ms of the default stream
        big.fill_(1.0)
    busy = torch.cuda.Event()
    busy.record()
    other = shim.Context(0)
    other.set_autotune(False)
    x, w, out = (T(other, t.shape, t.dtype, t.layout, _ptr=t.ptr) for t in (X, W, Y))
    other.memset(out.ptr, 255, out.nbytes)
    shim.device_conv2d(x, w, border_mode="half", out=out, flags=shim.NO_SLAB)
    assert other.last_variant == "tap pair cut"
    other.sync()
    assert not busy.query()                          # the default stream was busy all the while
    torch.cuda.synchronize()
    assert np.array_equal(y, out.to_host())
    other.close()
    ctx.close()


def test_a_replay_beside_other_launches():
    """A graph replayed on another context's stream counts the slices of its cut tiles for itself: beside launches of the context that captured it
    (and beside another graph's) every result is what it is alone."""
    a, b = shim.Context(0), shim.Context(0)
    for ctx in (a, b):
        ctx.set_autotune(False)
    X, W, Y, call = layer(a, np.float32)
    call()
    y = Y.to_host()
    outs = [T(a, Y.shape, np.float32, "nhwc") for _ in range(2)]
    graphs = []
    for out in outs:
        graphs.append(a.capture(lambda: [shim.device_conv2d(X, W, border_mode="half", out=out, flags=shim.NO_SLAB) for _ in range(3)]))
        assert a.last_variant == "tap pair cut"
    for _ in range(10):
        for t in outs + [Y]:
            a.memset(t.ptr, 255, t.nbytes)
        a.sync()
        for _ in range(5):
            b.check(b.lib.b200conv_graph_launch(b.h, graphs[0].h))
            graphs[1].launch()
            call()
        b.sync()
        a.sync()
        for t in outs + [Y]:
            assert np.array_equal(y, t.to_host())
    for g in graphs:
        g.destroy()
    b.close()
    a.close()
