"""Rules that the kernels' sources keep and that no result shows: what instructions ask of a warp."""
import os
import re

from theano_b200 import build

KERNELS = [f for f in build.SOURCES if f.startswith(("conv_", "wgrad_", "gemm_")) and f not in ("conv_reduce.cu", "conv_direct.cu")]


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(build.CSRC, name)).read())


def body(text, function):
    """What stands between the braces of a function."""
    start = text.index("{", re.search(r"\b%s\(" % function, text).end())
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError(function)


def test_accumulators_are_read_by_converged_warps():
    """tcgen05.ld.sync.aligned wants all lanes at once; the epilogues' loops send lanes without a pixel past the stores."""
    ptx = source("ptx.cuh")
    b = body(ptx, "void tmem_ld32")
    assert "tcgen05.ld.sync.aligned" in b and b.index("__syncwarp()") < b.index("asm")
    assert len(re.findall(r"tcgen05\.ld", ptx)) == 2 and not any("tcgen05.ld" in source(f) for f in KERNELS)
    users = [f for f in KERNELS if "tmem_ld16(" in source(f)]
    assert users == ["conv_cols.cu"]                  # there the caller brings the warp together
    sums = body(source("conv_cols.cu"), "void column_sums")
    assert sums.index("__syncwarp()") < sums.index("add_columns<") and source("conv_cols.cu").count("tmem_ld16(") == 1


def test_no_warp_leaves_others_at_a_named_barrier():
    """A named barrier waits without a bound.  Warps whose items end at one may not leave their loop when a wait runs out: the warps beside
    them may have seen that phase complete."""
    seen = []
    for f in KERNELS:
        text = source(f)
        if "named_barrier(" not in text:
            continue
        seen.append(f)
        assert "warp_wait_or_abort(" not in text, f
        for m in re.finditer(r"wait_or_walk_on\(", text):
            head = text.rindex("for (", 0, m.start())
            assert "ok" not in text[head:text.index("{", head)], (f, text[head:head + 120])
            assert "break" not in text[head:text.index("named_barrier(", m.start())].split("wait_or_walk_on", 1)[0], f
    assert seen == ["conv_slab.cu", "gemm_pair.cu", "conv_pair.cu", "conv_cols.cu", "wgrad_pair.cu"]
