"""Host-pointer calls: batches that travel in chunks of images, pageable and page-locked results, and the
pool of result memory."""
import gc

import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 7, 13, 24], ids=lambda n: "n%d" % n)     # one chunk, equal chunks, a smaller last one
@pytest.mark.parametrize("pageable_out", [False, True])
def test_chunked_batches_against_oracle(n, pageable_out):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(n)
    x = rs.standard_normal((n, 64, 61, 64)).astype(np.float32)              # 1 MB per image and side
    w = (rs.standard_normal((64, 64, 1, 1)) / 8).astype(np.float32)
    b, r = rs.standard_normal(64).astype(np.float32), rs.standard_normal(x.shape).astype(np.float32)
    kw = dict(border_mode="valid", subsample=(1, 1))
    out = np.full(x.shape, 7, np.float32) if pageable_out else None
    y = shim.conv2d_forward(x, w, bias=b, residual=r, out=out, ctx=ctx, **kw)
    assert (y is out) == pageable_out
    # TF32 rounds each factor by at most 2^-10 relative: 5e-3 of the largest result is the repository's bound
    assert O.rel_err(y, O.conv2d(x, w, **kw) + b[None, :, None, None] + r) < 5e-3
    out = np.full(x.shape, 7, np.float32) if pageable_out else None
    dx = shim.conv2d_grad_inputs(w, r, x.shape[2:], out=out, ctx=ctx, **kw)
    assert O.rel_err(dx, O.conv2d_grad_inputs(w, r, x.shape[2:], **kw)) < 5e-3
    # results of one call are inputs of the next: page-locked inputs take no staging copy
    dw = shim.conv2d_grad_weights(y, dx, (1, 1), ctx=ctx, **kw)
    assert O.rel_err(dw, O.conv2d_grad_weights(np.array(y), np.array(dx), (1, 1), **kw)) < 5e-3


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 13], ids=lambda n: "n%d" % n)
def test_chunked_batches_in_page_locked_memory(n):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(n)
    x, y, dx = (ctx.pinned_empty((n, 64, 61, 64), np.float32) for _ in range(3))
    x[...] = rs.standard_normal(x.shape)
    w = (rs.standard_normal((64, 64, 1, 1)) / 8).astype(np.float32)
    kw = dict(border_mode="valid", subsample=(1, 1))
    assert shim.conv2d_forward(x, w, out=y, ctx=ctx, **kw) is y
    assert O.rel_err(np.array(y), O.conv2d(np.array(x), w, **kw)) < 5e-3      # TF32 rounds each factor by at most 2^-10
    assert shim.conv2d_grad_inputs(w, x, out=dx, ctx=ctx, **kw) is dx
    assert O.rel_err(np.array(dx), O.conv2d_grad_inputs(w, np.array(x), x.shape[2:], **kw)) < 5e-3


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [1, 30], ids=["filters", "residual"])
def test_small_inputs_wait_for_large_ones_in_their_own_slot(extra):
    """Small inputs share a slot of the staging ring; an image of more than the whole ring must not take it."""
    ctx = shim.get_context(0)
    rs = np.random.RandomState(1)
    n, c, h, w = 1, 8 if extra == 1 else 1, 1200, 1300                      # 50 MB in, or 6 MB in and a residual
    k = 1 if extra == 1 else 8
    # small whole numbers: products and sums are exact in TF32
    x = rs.randint(-8, 9, (n, c, h, w)).astype(np.float32)
    f = rs.randint(-8, 9, (k, c, 1, 1)).astype(np.float32)
    b = rs.randint(-8, 9, k).astype(np.float32)
    r = None if extra == 1 else rs.randint(-8, 9, (n, k, h, w)).astype(np.float32)
    y = shim.conv2d_forward(x, f, bias=b, residual=r, ctx=ctx)
    want = np.einsum("kc,nchw->nkhw", f[:, :, 0, 0], x) + b[None, :, None, None] + (0 if r is None else r)
    assert np.array_equal(y, want)


@pytest.mark.gpu
@pytest.mark.parametrize("page_locked", [False, True])
@pytest.mark.parametrize("start,c", [(0, 64), (0.25, 64), (1, 64), (0, 128)], ids=["front", "inside", "back", "same"])
def test_a_result_may_lie_over_the_input(start, c, page_locked):
    """The memory of out= holds the input: a batch in chunks would overwrite images that have not gone up yet."""
    ctx = shim.get_context(0)
    rs = np.random.RandomState(5)
    n, k, h = 16, 128, 64                                                    # 2 MB per image of the result, as much or half of the input
    w = (rs.standard_normal((k, c, 1, 1)) / 8).astype(np.float32)
    v = np.ascontiguousarray(w.transpose(1, 0, 2, 3))
    kw = dict(border_mode="valid", subsample=(1, 1))
    x = rs.standard_normal((n, c, h, h)).astype(np.float32)
    for call, want in ((lambda a, o: shim.conv2d_forward(a, w, out=o, ctx=ctx, **kw), O.conv2d(x, w, **kw)),
                       (lambda a, o: shim.conv2d_grad_inputs(v, a, out=o, ctx=ctx, **kw), O.conv2d_grad_inputs(v, x, (h, h), **kw))):
        out = ctx.pinned_empty((n, k, h, h), np.float32) if page_locked else np.empty((n, k, h, h), np.float32)
        first = int(start * (out.size - x.size))
        a = out.reshape(-1)[first:first + x.size].reshape(x.shape)
        a[...] = x
        assert np.shares_memory(a, out)
        got = call(a, out)
        assert got is out and O.rel_err(got, want) < 5e-3      # TF32 rounds each factor by at most 2^-10 relative


@pytest.mark.gpu
def test_host_calls_without_a_staging_ring(monkeypatch):
    """No copy threads, or no page-locked memory for the ring: small and large arrays travel the driver's way."""
    monkeypatch.setenv("B200CONV_COPY_THREADS", "0")
    ctx = shim.Context(0)
    rs = np.random.RandomState(2)
    kw = dict(border_mode="half", subsample=(1, 1))
    for n, h in ((2, 9), (12, 96)):                          # 3 KB, and 14 MB in chunks
        x = rs.standard_normal((n, 32, h, h)).astype(np.float32)
        w = (rs.standard_normal((32, 32, 3, 3)) / 17).astype(np.float32)
        out = np.full(x.shape, 7, np.float32)
        assert O.rel_err(shim.conv2d_forward(x, w, out=out, ctx=ctx, **kw), O.conv2d(x, w, **kw)) < 5e-3
        assert O.rel_err(shim.conv2d_grad_inputs(w, x, ctx=ctx, **kw), O.conv2d_grad_inputs(w, x, (h, h), **kw)) < 5e-3
        assert O.rel_err(shim.conv2d_grad_weights(x, x, (3, 3), ctx=ctx, **kw), O.conv2d_grad_weights(x, x, (3, 3), **kw)) < 5e-3
    ctx.close()


@pytest.mark.gpu
def test_a_capture_refuses_host_calls_and_leaves_the_staging_ring_alone():
    """An event of the ring recorded in a capture could not be waited for by the calls that come after it."""
    ctx = shim.Context(0)
    x = np.arange(2 * 3 * 8 * 8, dtype=np.float32).reshape(2, 3, 8, 8)
    w, want = np.ones((5, 3, 1, 1), np.float32), x.reshape(2, 3, 4, 2, 4, 2).max(axis=(3, 5))
    y = shim.maxpool2x2(x, ctx=ctx)
    for call in (lambda: shim.maxpool2x2(x, ctx=ctx), lambda: shim.maxpool2x2_grad(x, y, y, ctx=ctx), lambda: shim.conv2d_forward(x, w, ctx=ctx)):
        with pytest.raises(ValueError, match="cannot be captured"):
            ctx.capture(call)
    for _ in range(40):                          # more calls than the ring has slots
        assert np.array_equal(shim.maxpool2x2(x, ctx=ctx), want)
    ctx.close()


@pytest.mark.gpu
def test_results_keep_their_values_while_others_are_made():
    ctx = shim.get_context(0)
    rs = np.random.RandomState(0)
    xs = [rs.standard_normal((8, 8, 40, 40)).astype(np.float32) for _ in range(6)]
    ys = [shim.maxpool2x2(x, ctx=ctx) for x in xs]
    for x, y in zip(xs, ys):
        assert np.array_equal(y, x.reshape(8, 8, 20, 2, 20, 2).max(axis=(3, 5)))


class _FakeLibrary(object):
    """Stands in for the library's page-locked allocator."""

    def __init__(self):
        self.made, self.buffers = 0, {}

    def b200conv_host_alloc(self, h, size, p):
        buf = np.empty(size, np.uint8)
        self.buffers[buf.ctypes.data] = buf
        p._obj.value = buf.ctypes.data
        self.made += 1
        return 0

    def b200conv_host_free(self, h, p):
        del self.buffers[p.value]
        return 0


def test_result_pool_reuses_and_gives_back(monkeypatch):
    class Ctx(object):
        lib, h = _FakeLibrary(), None
    monkeypatch.setattr(shim, "load_library", lambda: Ctx.lib)
    pool = shim._ResultPool()
    pool.LIMIT, pool.KEEP = 4 << 20, 1 << 20
    f32 = np.dtype(np.float32)
    assert pool.empty(Ctx, (10,), f32).base is None                     # small: an ordinary array
    a = pool.empty(Ctx, (100, 1000), f32)
    ptr = a.ctypes.data
    view = a[3:5]
    del a
    gc.collect()
    assert pool.kept == 0                                               # the view keeps the memory
    del view
    b = pool.empty(Ctx, (99, 1001), f32)
    assert b.ctypes.data == ptr and b.shape == (99, 1001) and b.dtype == f32 and b.flags.writeable
    many = [pool.empty(Ctx, (1 << 18,), f32) for _ in range(8)]         # 1 MB each: over the limit
    assert sum(m.base is not None for m in many) == 3 and pool.total <= pool.LIMIT
    del many, b
    gc.collect()
    assert pool.kept <= pool.KEEP and pool.total == pool.kept and len(Ctx.lib.buffers) <= 2
    pool.trim()                                                         # nothing is out: all of it goes back
    assert pool.total == pool.kept == 0 and not Ctx.lib.buffers


def _pool(monkeypatch, limit=None):
    class Ctx(object):
        lib, h = _FakeLibrary(), None
    monkeypatch.setattr(shim, "load_library", lambda: Ctx.lib)
    pool = shim._ResultPool()
    if limit is not None:
        pool.LIMIT = pool.KEEP = limit
    return pool, Ctx


def _passes(pool, ctx, sizes, count):
    """Page-locked allocations of each of `count` passes that hold results of `sizes` bytes and then drop them."""
    made = []
    for _ in range(count):
        before = ctx.lib.made
        held = [pool.empty(ctx, (n,), np.dtype(np.uint8)) for n in sizes]
        assert pool.total <= pool.LIMIT
        made.append(ctx.lib.made - before)
        del held
        gc.collect()
    return made


@pytest.mark.parametrize("sizes", [[300 << 20], [90 << 20, 100 << 20, 110 << 20], [6 << 20] * 60, [26 << 20, 26 << 20, 1 << 20]],
                         ids=["one", "three", "sixty", "training"])
def test_result_pool_does_not_lock_memory_again_and_again(monkeypatch, sizes):
    """Page-locking costs more than an ordinary array: once per block, and never on every pass."""
    pool, ctx = _pool(monkeypatch)
    made = _passes(pool, ctx, sizes, 12)
    assert not any(made[8:]), made
    if sum(sizes) < pool.LIMIT:                                          # all of them end up in locked memory
        assert all(pool.empty(ctx, (n,), np.dtype(np.uint8)).base is not None for n in sizes)
    # what is locked was earned: its bytes went out as ordinary arrays, beyond the credit at the start
    assert pool.total <= pool.CREDIT + 12 * sum(sizes)
    assert _passes(pool, ctx, [1 << 29], 2) == [0, 0]                    # beyond the limit: ordinary


def test_result_pool_gives_unused_sizes_back(monkeypatch):
    pool, ctx = _pool(monkeypatch)
    _passes(pool, ctx, [150 << 20], 6)
    assert pool.kept >= 150 << 20
    made = _passes(pool, ctx, [6 << 20] * 20, 20)
    assert not any(made[14:]) and pool.total <= 256 << 20 and sum(made) == 20
    assert len(ctx.lib.buffers) == 20 and pool.total == pool.kept


def test_result_pool_does_not_follow_sizes_that_keep_changing(monkeypatch):
    pool, ctx = _pool(monkeypatch)
    pool.STALE = 4
    made = [sum(_passes(pool, ctx, [n << 20], 1)) for _ in range(10) for n in (20, 24, 32, 40, 48, 64, 96, 128)]
    assert sum(made) <= 3                                                # the credit at the start, and never again


def test_result_pool_can_be_turned_off(monkeypatch):
    pool, ctx = _pool(monkeypatch, 0)
    a = pool.empty(ctx, (1 << 20,), np.dtype(np.float32))
    assert a.flags.owndata and ctx.lib.made == 0


def test_operands_in_the_other_byte_order_are_converted():
    a, b = np.arange(6, dtype=">f4"), np.arange(4, dtype=">f4")
    for v, w in zip(shim._common(a, b), (a, b)):
        assert v.dtype.isnative and v.dtype == np.float32 and np.array_equal(v, w)
