"""Bounds-checked build: every access of the fixed-point kernels to their matrices stays inside what the matrix has
(writes) or may be read beside it (lanes without work), in every launch shape; and the FP64 kernels of the entry points
that start in fixed point are still checked."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def cases(cuda):
    from tokura_zgeev_batched_gb300 import build

    build.build(debug=True)
    env = dict(os.environ, TOKURA_ZGEEV_DEBUG_BOUNDS="1")
    res = subprocess.run([sys.executable, os.path.join(HERE, "debug_bounds_fixed_run.py")], env=env,
                         capture_output=True, text=True, timeout=900)
    assert res.returncode == 0, res.stderr[-4000:]
    return json.loads(res.stdout.strip().splitlines()[-1])


def test_no_access_outside(cases):
    bad = {k: v for k, v in cases.items() if v["violations"] != 0}
    assert len(cases) >= 60 and not bad, bad


def test_the_fixed_point_kernels_are_checked(cases):
    """Thousands of checked accesses to a matrix in every call that starts in fixed point, none in the others."""
    for name, case in cases.items():
        if "FP64" in name:
            assert case["checks"] == 0, name
        else:
            assert case["checks"] > 1000, name


def test_the_release_library_counts_nothing():
    from tokura_zgeev_batched_gb300 import api

    assert api.lib().tokuraDebugChecks(None) == -2
