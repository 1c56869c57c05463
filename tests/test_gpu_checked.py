"""The parity suites against the bounds-checked library (librppb_checked.so).

In that library every global load and store of the kernels is checked against the device regions of
the call that launched it, and a call with an access outside them returns an error status
(include/rppb_frontend.h, rpp_b200/csrc/check.cu).  Running the parity suites against it in a child
process (RPPB_LIBRARY=checked) shows that every kernel stays inside the caller's tensors as their
descriptors describe them, the per-sample tensors, the workspace and the handle's tables, on every
case those suites cover, with the same outputs; tests/test_gpu_checked_fuzz.py adds seeded random valid
calls of every entry point.  tests/test_gpu_checked_hooks.py, run in the same child process, shows that
the checks do fire.  Outside this check: the tensor-core kernels' TMA loads
(their reach is bounded by the tensor maps, which the driver validates), and the serving thread's
copy kernels, which run outside any call.  Tests of time are left out; the only tests that may skip are
those against the reference's own host library, where that is not built.
"""
import os
import re
import subprocess
import sys

import pytest

from oracle import reference_lib_path
from rpp_b200 import lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SUITES = ["tests/test_gpu_ops.py", "tests/test_gpu_normalize_nd.py", "tests/test_gpu_frontend.py",
          "tests/test_gpu_frontend_tc.py", "tests/test_gpu_tc.py", "tests/test_gpu_parity_reference.py",
          "tests/test_gpu_edges.py", "tests/test_gpu_parity_fuzz.py", "tests/test_gpu_nsr_intervals.py",
          "tests/test_gpu_resample_held.py", "tests/test_gpu_spectrogram_tiles.py", "tests/test_gpu_ragged_batches.py",
          "tests/test_gpu_normalize_rows.py", "tests/test_gpu_frontend_128.py",
          "tests/test_gpu_checked_hooks.py", "tests/test_gpu_checked_fuzz.py"]
TIMED = "spread_over_the_gpu or keep_their_time"


@pytest.mark.gpu
def test_parity_suites_under_the_checked_library():
    assert os.path.isfile(lib.CHECKED_LIB_PATH), "build it with `python -m rpp_b200.build --checked`"
    env = dict(os.environ, RPPB_LIBRARY="checked")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-rs", "-m", "gpu", "-k", f"not ({TIMED})", "-p",
                        "no:cacheprovider"] + SUITES, cwd=ROOT, env=env, capture_output=True, text=True, timeout=1800)
    tail = r.stdout[-4000:] + r.stderr[-2000:]
    assert r.returncode == 0, tail
    last = r.stdout.splitlines()[-1]
    skipped = re.findall(r"^SKIPPED \[(\d+)\] [^:]+:\d+: (.*)$", r.stdout, re.M)
    if os.path.isfile(reference_lib_path()):
        assert not skipped, tail
    assert all("reference host library not built" in reason for _, reason in skipped), tail
    total = re.search(r"(\d+) skipped", last)
    assert " passed" in last and int(total[1] if total else 0) == sum(int(k) for k, _ in skipped), tail
