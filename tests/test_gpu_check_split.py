"""The bounds checks of the split in the -DGQS_CHECK build: the tests of its paths, of what it leaves and of its scratch, run by
that build in a child process, find no violation (a violation is a status, which they would report)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

TESTS = os.path.dirname(os.path.abspath(__file__))


def test_check_build_finds_no_violation_in_the_split():
    import build_lib
    lib = build_lib.build(check=True)["lib"]
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider"]
                       + [os.path.join(TESTS, f) for f in ("test_gpu_split.py", "test_gpu_leftovers.py", "test_gpu_split_scratch.py")],
                       env=dict(os.environ, GQS_LIB=lib), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:]
    assert " passed" in r.stdout
