"""The pairwise kernels, the ordering and the ensemble plans on the bounds-checked build: their items (rows, j tiles,
slabs), table records and ordering indices at the sizes where groups, chunks, tiles and bricks end, and with positions
that are not finite."""
import os
import re
import subprocess
import sys

import pytest

import steps_gb300 as S

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = [
    "tests/test_gpu_sym.py::test_r3_sizes",
    "tests/test_gpu_sym.py::test_r3_softened_and_coincident",
    "tests/test_gpu_sym.py::test_periodic_sizes",
    "tests/test_gpu_sym.py::test_periodic_hard_decisions",
    "tests/test_gpu_sym.py::test_t3_brick_records",
    "tests/test_gpu_sym.py::test_tables_that_are_not_odd",
    "tests/test_gpu_sym.py::test_fp64_sizes",
    "tests/test_gpu_shapes.py::test_r3",
    "tests/test_gpu_shapes.py::test_ordering_sizes",
    "tests/test_gpu_shapes.py::test_radix_ordering_sizes",
    "tests/test_gpu_ensemble.py::test_every_plan",
    "tests/test_gpu_nonfinite.py",
]


@pytest.mark.skipif(os.environ.get("STEPS_GB300_LIB") == S.CHECK_LIB_PATH,
                    reason="already running on the bounds-checked library")
def test_pairwise_cases_under_bounds_checks():
    assert os.path.exists(S.CHECK_LIB_PATH), "build() makes the bounds-checked library"
    env = dict(os.environ, STEPS_GB300_LIB=S.CHECK_LIB_PATH, STEPS_GB300_QUIET="1")
    cmd = [sys.executable, "-m", "pytest", "-q", "-m", "gpu", "-p", "no:cacheprovider", "-x", *CASES]
    r = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True, timeout=1200)
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-2000:]
    m = re.search(r"(\d+) passed", r.stdout)
    assert m and int(m.group(1)) >= len(CASES) and "failed" not in r.stdout, r.stdout[-2000:]
