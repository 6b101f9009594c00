"""Kernels launched while the grid before them still runs (programmatic dependent launch) read what that grid
writes: none of their pointers may be declared read-only for the kernel's lifetime, since such loads need not be
coherent and may be moved above griddepcontrol.wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "shll-sve-cfd_gb300", "csrc")


def chained_kernels():
    """(name, parameters, body) of every kernel whose body waits for the grid before it."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(([^{;]*?)\)\s*\{(.*?)\n\}", text, re.S):
            if re.search(r"griddepcontrol\.wait|after_previous_step\(\)", m.group(3)):
                found.append(m.groups())
    return found


def test_chained_kernels_have_no_read_only_pointers():
    kernels = chained_kernels()
    assert {"k_step2", "k_step2d", "k_step2d2", "k_step2d_o2"} <= {k[0] for k in kernels}
    for name, params, body in kernels:
        assert "__restrict__" not in params, name
        assert "__ldg" not in body, name
