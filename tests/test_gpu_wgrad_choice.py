"""Which gradWeights kernel runs: what a context reports, and what the flags that ask for a kernel or bar one do on a context that
other calls have used, with timing on."""
import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import shim

pytestmark = pytest.mark.gpu
DTYPES = pytest.mark.parametrize("dtype", [np.float32, np.float16], ids=["f32", "f16"])
ROWS, NO_ROWS, NO_GROUP = shim.ROWS, shim.NO_ROWS, shim.NO_GROUP
KERNELS = ("wgrad tap", "wgrad groups", "wgrad rows")        # by the number in tuning files


def _layer(ctx, dtype, xs, k, ks, s=1, g=1):
    """run(flags) -> variant, on operands of values -1, 0, 1: sums are whole numbers that both types hold."""
    kw = dict(border_mode="half", subsample=(s, s), num_groups=g)
    rs = np.random.RandomState(k + ks)
    x = rs.randint(-1, 2, xs).astype(dtype)
    ho, wo = O.conv2d(np.zeros((1, g) + xs[2:], np.float32), np.zeros((g, 1, ks, ks), np.float32), **kw).shape[2:]
    dy = rs.randint(-1, 2, (xs[0], k, ho, wo)).astype(dtype)
    want = O.conv2d_grad_weights(x.astype(np.float32), dy.astype(np.float32), (ks, ks), **kw).astype(dtype)
    X, DY = shim.DeviceTensor.from_host(ctx, x, "nhwc"), shim.DeviceTensor.from_host(ctx, dy, "nhwc")

    def run(flags=0):
        got = shim.device_grad_weights(X, DY, (ks, ks), flags=flags, **kw).to_host()
        assert np.array_equal(got, want)
        return ctx.last_variant
    return run


@DTYPES
def test_reported_variant(dtype):
    ctx = shim.Context(0)
    narrow = _layer(ctx, dtype, (2, 32, 14, 14), 24, 3)
    wide = _layer(ctx, dtype, (2, 256, 7, 7), 256, 3)
    stem = _layer(ctx, dtype, (2, 3, 30, 30), 100, 3)
    assert narrow(ROWS) == "wgrad rows"
    assert wide(NO_GROUP) == "wgrad pair"
    assert narrow(ROWS) == "wgrad rows"
    assert stem() == "wgrad tap"
    assert narrow(NO_GROUP) == "wgrad tap"
    ctx.set_autotune(False)
    assert narrow(NO_ROWS) == "wgrad groups"
    ctx.close()


@DTYPES
@pytest.mark.parametrize("xs,k,ks", [((2, 32, 28, 28), 32, 3), ((16, 64, 14, 14), 30, 5), ((4, 100, 9, 30), 20, 2), ((8, 20, 40, 40), 128, 3)])
def test_reported_variant_is_the_remembered_one(tmp_path, dtype, xs, k, ks):
    ctx = shim.Context(0)
    run = _layer(ctx, dtype, xs, k, ks)
    first = run()
    ctx.tuning_save(str(tmp_path / "tuning"))
    choices = [l.split() for l in open(str(tmp_path / "tuning")).read().splitlines()]
    (choice,) = [KERNELS[int(l[2])] for l in choices if l[0] == "a" and l[1].startswith("4.")]
    assert first == choice and run() == choice
    ctx.close()


FORMS = {"plain": ((4, 32, 14, 14), 24, 3, 1, 1), "groups": ((64, 256, 28, 28), 256, 3, 1, 32), "folded": ((64, 3, 32, 32), 32, 3, 1, 1),
         "blocks": ((64, 3, 64, 64), 24, 7, 2, 1)}


@DTYPES
@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("first", [NO_ROWS, NO_GROUP, ROWS, 0], ids=["NO_ROWS", "NO_GROUP", "ROWS", "none"])
def test_flags_hold_for_their_call_only(dtype, form, first):
    """Whatever the first call asked for, each later one gets what its own flags say."""
    ctx = shim.Context(0)
    run = _layer(ctx, dtype, *FORMS[form])
    run(first)
    for _ in range(2):
        assert run(NO_ROWS) != "wgrad rows"
        assert run(ROWS) == "wgrad rows"
        assert run(NO_GROUP) == "wgrad tap"
        assert run(NO_ROWS | ROWS) != "wgrad rows"
        assert run(NO_GROUP | ROWS) == "wgrad rows"
        assert run(NO_GROUP | NO_ROWS) == "wgrad tap"
        chosen = run()
        assert run() == chosen
        if form == "groups":         # 83 against 180 us in float32, 256 images: no close call
            assert chosen == "wgrad rows"
    ctx.close()


@DTYPES
def test_rows_flag_where_the_kernel_does_not_apply(dtype):
    ctx = shim.Context(0)
    run = _layer(ctx, dtype, (2, 24, 12, 12), 100, 3)
    chosen = run()
    assert chosen in ("wgrad tap", "wgrad groups") and run(ROWS) == run() == chosen
    assert run(ROWS | NO_GROUP) == "wgrad tap"
    ctx.close()


@pytest.mark.parametrize("tuned", [True, False])
@pytest.mark.parametrize("dtype,n,kind", [(np.float32, 49, "wgrad tap"), (np.float32, 50, "wgrad rows"), (np.float16, 199, "wgrad tap"),
                                          (np.float16, 200, None), (np.float16, 1000, "wgrad rows")])
@pytest.mark.parametrize("xs,k,ks,s", [((3, 10, 10), 32, 3, 1), ((2, 20, 20), 16, 3, 2)], ids=["folded", "blocks"])
def test_layers_with_few_channels(dtype, tuned, n, kind, xs, k, ks, s):
    """100 output pixels per image: below and above the lines of the rule; None: between them, where a first call with timing on decides."""
    ctx = shim.Context(0)
    ctx.set_autotune(tuned)
    run = _layer(ctx, dtype, (n,) + xs, k, ks, s)
    first = run()
    assert run() == first == (kind or (first if tuned else "wgrad rows"))
    assert first in ("wgrad tap", "wgrad rows")
    ctx.close()


@pytest.mark.parametrize("dtype,n,kind", [(np.float32, 1, "wgrad rows"), (np.float16, 59, "wgrad groups"), (np.float16, 60, "wgrad rows")])
def test_merged_groups_without_timing(dtype, n, kind):
    ctx = shim.Context(0)
    ctx.set_autotune(False)
    assert _layer(ctx, dtype, (n, 64, 10, 10), 64, 3, g=8)() == kind
    ctx.close()


def test_a_file_of_other_kernels_is_not_loaded(tmp_path):
    """Choices timed on other kernels would keep this version's from being tried."""
    path = str(tmp_path / "tuning")
    ctx = shim.Context(0)
    _layer(ctx, np.float32, (2, 32, 14, 14), 24, 3)()
    ctx.tuning_save(path)
    head, rest = open(path).read().split("\n", 1)
    assert " kernels " in head and ctx.tuning_load(path) == len(rest.splitlines()) > 0
    older = head[:head.index(" kernels ")]                       # as files before that number have it
    for other in (older, older + " kernels 1", head + "1"):
        open(path, "w").write(other + "\n" + rest)
        with pytest.raises(ValueError, match="version of the kernels"):
            ctx.tuning_load(path)
    ctx.close()
