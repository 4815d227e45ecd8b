"""The kernels are launched while the kernel before them may still be writing, and wait
for it at their start.  A non-coherent load (__ldg, ld.global.nc, a const __restrict__
pointer) may be moved above that wait and is only defined for memory that nobody writes
while the kernel lives: the sources hold none."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_non_coherent_loads_in_the_kernels():
    files = glob.glob(os.path.join(ROOT, "sph-2d_b200", "csrc", "*.cu*"))
    assert len(files) >= 8
    for f in files:
        code = re.sub(r"//[^\n]*", "", open(f).read())
        assert not re.search(r"__ldg\b|\bld\.global(\.\w+)*\.nc\b|__restrict__", code), f
