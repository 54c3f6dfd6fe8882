"""The range-checked build runs the tests of the columns kernel, the per-tap kernel on pairs with its cut tiles, tile widths and filter packing:
every store of theirs, slab index and tiled store lies inside of its buffer."""
import os
import subprocess
import sys

import pytest

from theano_b200 import build as lib_build

pytestmark = pytest.mark.gpu
FILES = ["test_gpu_columns.py", "test_gpu_stem_gradient.py", "test_gpu_tap_pairs.py", "test_gpu_cut_tiles.py", "test_gpu_tile_widths.py", "test_gpu_filter_packing.py"]


@pytest.mark.parametrize("name", FILES)
def test_range_checked_build_passes(name):
    if not os.path.exists(lib_build.DEBUG_LIB):
        pytest.skip("libb200conv_debug.so is not built (python -m theano_b200.build --debug)")
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider", os.path.join(here, name)],
                       cwd=os.path.dirname(here), env=dict(os.environ, B200CONV_LIB=lib_build.DEBUG_LIB), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
