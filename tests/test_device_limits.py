"""A kernel's shared-memory limit belongs to a device, and a process may hold contexts on several: no limit is raised from the
initialiser of a static variable, which runs once, on whatever device is current then (needs no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-quicksort_gb300", "csrc")


def test_no_limit_is_raised_once_per_process():
    raised = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        raised += text.count("cudaFuncSetAttribute")
        for m in re.finditer(r"\bstatic\b[^;{}()]*=\s*\[", text):  # static ... = [] { ... }()
            body = text[m.start():text.index("}()", m.start())]
            assert "allow_smem" not in body and "cudaFuncSetAttribute" not in body, (name, body)
    assert raised >= 2  # the kernel variants' and the split's
