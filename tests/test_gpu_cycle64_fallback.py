"""The FP64 V-cycle on devices that cannot place a cluster of 16 blocks: side 33
colour-split, restricted into and prolongated from the one-block tail of side 17, bit for
bit with its operators (the tests of test_gpu_cycle64.py in the checked build, which takes
that form on every device)."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r'''
import ctypes, sys
import pytest
sys.path.insert(0, ROOT)
from mojo_poissonrecon_b200 import _native
L = _native.lib()
assert L.pb_checked_build() == 1
doubles, flags = ctypes.c_int64(), ctypes.c_int64()
assert L.pb_vcycle_level_size(33, ctypes.byref(doubles), ctypes.byref(flags)) == 0
assert flags.value > 0 and doubles.value > 33 ** 3  # by colour, not the cluster's dense grid
assert L.pb_vcycle_level_size(17, ctypes.byref(doubles), ctypes.byref(flags)) == 0 and flags.value == 0
status = pytest.main(["-q", "-x", "-p", "no:cacheprovider", ROOT + "/tests/test_gpu_cycle64.py"])
assert status == 0 and _native.check_word() == 0
print("fallback ok")
'''


def test_cycles_match_their_operators_without_a_cluster():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import buildlib

    if not os.path.exists(buildlib.CHECKED_LIBRARY):
        pytest.skip("checked library not built")
    proc = subprocess.run([sys.executable, "-c", SCRIPT.replace("ROOT", repr(ROOT))], cwd=ROOT, capture_output=True,
                          text=True, timeout=600, env=dict(os.environ, MPR_B200_CHECKED="1"))
    assert proc.returncode == 0 and "fallback ok" in proc.stdout, (proc.stdout + proc.stderr)[-3000:]
