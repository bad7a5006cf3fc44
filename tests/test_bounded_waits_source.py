"""The wait that the barrier test makes run out is the wait that the persistent
peel uses, and there is no other grid barrier in the library."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tdtdecomposition_gb300", "csrc")


def _kernel(src, name):
    at = re.search(r"__global__[^;{]*\b%s\(" % name, src).start()
    return src[at:src.index("\n}\n", at)]


def test_probe_waits_in_the_peels_barrier():
    src = open(os.path.join(CSRC, "peel.cu")).read()
    probe, peel = (_kernel(src, k) for k in ("barrier_probe_kernel", "peel_kernel"))
    assert "round_barrier(" in probe and "round_barrier(" in peel
    defined = [m for f in glob.glob(os.path.join(CSRC, "*.cu*"))
               for m in re.findall(r"__device__[^;{]*\bbool (\w*barrier\w*)\(", open(f).read())]
    assert defined == ["round_barrier"]
