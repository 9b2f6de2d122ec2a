"""When a small sort's counters are cleared (gpu-quicksort_gb300/csrc/gqs_counters.h), on the CPU: after a launch that failed
halfway, in new scratch, and not again once they are zero."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_counters_are_zero_for_every_sort(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "counters_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "gpu-quicksort_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "counters_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
