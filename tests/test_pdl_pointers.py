"""Kernels launched programmatically behind their predecessor read what it
writes while both are resident.  A pointer declared __restrict__ lets the
compiler take a load of it for one that no wait or memory clobber can change
(and, with const, use the read-only cache), so those kernels declare none."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-montecarlo-risk_gb300", "csrc")


def test_kernels_that_wait_for_their_predecessor_restrict_no_pointer():
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for kernel in text.split("__global__")[1:]:
            m = re.search(r"(\w+_kernel)\s*\(([^{;]*)\)\s*\{", kernel)
            body = kernel[m.end():kernel.find("\n}", m.end())] if m else ""
            if "pdl_enter()" in body or "griddepcontrol.wait" in body:
                found[m.group(1)] = m.group(2), body
    assert set(found) >= {"chol_step_kernel", "chol_panel_kernel", "chol_finish_kernel"}, set(found)
    assert not [name for name, (args, body) in found.items() if "__restrict__" in args or "__ldg" in body]
