"""CPU: every kernel that pdl_launch starts waits for the grid before it
(pdl_entry) before it does anything else: with the programmatic-serialisation
attribute a kernel without the wait would read its inputs while they are
written."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "alamo_gb300", "csrc")


def test_kernels_launched_dependently_wait_first():
    src = "".join(re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    launched = set(re.findall(r"pdl_launch\(\s*(k_\w+)", src))
    assert len(launched) >= 15, launched
    for name in sorted(launched):
        bodies = re.findall(r"\b%s\s*\([^;{]*\)\s*\{\s*([^;]*;)" % name, src)
        assert bodies, name
        for first in bodies:
            assert first.strip() == "pdl_entry();", (name, first)
