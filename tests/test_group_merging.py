"""How gradWeights merges the groups of grouped layers: the rule is compiled from the library's own header and
enumerated on the CPU, and layers whose largest merge is not aligned run on the GPU against the oracle."""
import os
import subprocess

import numpy as np
import pytest

from oracle import corr_oracle as O
from theano_b200 import build, shim

PROGRAM = r"""
#include <stdio.h>
#include "geometry.h"
using namespace b200;
// Every layer that runs with the groups merged as for the other directions, or unmerged, has to run here too.
int main() {
  long long lost = 0, seen = 0, outside = 0;
  for (int dtype = 0; dtype < 2; ++dtype)
    for (int g = 2; g <= 1024; g = g < 64 ? g + 1 : g + 4)
      for (int cg = 1; cg <= 64 && cg * g <= 2048; ++cg)
        for (int kg = 1; kg <= 256 && kg * g <= 4096; kg = kg < 128 ? kg + 1 : kg + 4) {
          b200conv_desc d = {2, cg * g, 9, 9, kg * g, 3, 3, 9, 9, 1, 1, 1, 1, 1, 1, 1, 1, g, 0, dtype};
          const int f = merge_factor(d), m = merge_factor_wgrad(d);
          if (g % m) ++outside;
          if (!umma_ok(d) && !(f > 1 && umma_ok(merged_groups(d, f)))) continue;
          ++seen;
          const bool runs = umma_ok(d) || (m > 1 && umma_ok(merged_groups(d, m)));
          if (!runs && lost++ < 5) fprintf(stderr, "lost: dtype %d groups %d Cg %d Kg %d (m = %d)\n", dtype, g, cg, kg, m);
        }
  printf("%lld %lld %lld\n", seen, lost, outside);
  return 0;
}
"""


def test_no_grouped_layer_is_lost(tmp_path):
    src, exe = tmp_path / "merge.cpp", tmp_path / "merge"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)])
    seen, lost, outside = map(int, subprocess.check_output([str(exe)]).split())
    assert seen > 50000 and lost == 0 and outside == 0


# the largest divisor within 128 x 128 leaves pieces that are not whole 16 bytes; or no divisor fits 128 filters
UNALIGNED = [(np.float32, 816, 816, 816), (np.float32, 196, 196, 196), (np.float16, 280, 280, 280), (np.float16, 8, 160, 2),
             (np.float16, 144, 24, 6), (np.float32, 4, 200, 2), (np.float16, 32, 1024, 32)]


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("dtype,c,k,g", UNALIGNED, ids=lambda v: getattr(v, "__name__", str(v)))
def test_grad_weights_of_unaligned_merges(dtype, c, k, g, layout):
    ctx = shim.get_context(0)
    rs = np.random.RandomState(g)
    x, dy = (rs.standard_normal((3, n, 11, 9)).astype(dtype) for n in (c, k))
    kw = dict(border_mode="half", num_groups=g)
    f = np.float32
    want = O.conv2d_grad_weights(x.astype(f), dy.astype(f), (3, 3), **kw)
    X, DY = (shim.DeviceTensor.from_host(ctx, a, layout) for a in (x, dy))
    tol = 5e-3 if dtype == np.float32 else 2e-2          # the repository's bounds: TF32 factors, float16 tensors
    got = shim.device_grad_weights(X, DY, (3, 3), flags=shim.FORCE_UMMA, **kw)
    assert O.rel_err(got.to_host().astype(f), want) < tol
    full = shim.DeviceTensor(ctx, want.shape, f)
    shim.device_grad_weights(X, DY, (3, 3), out=full, **kw)      # float32 gradient of float16 tensors
    assert ctx.last_algo == "umma" and O.rel_err(full.to_host(), want) < tol
