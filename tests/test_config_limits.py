"""Configurations with an infinite support are refused, and at once: the search for the
support's bound on the squared distance has no end there.  In a child process with a
time limit, through the pair search for callers with their own buffers, which checks
the configuration before it looks for a device (no buffer is touched)."""
import subprocess
import sys

import pytest

import sph_b200 as S

CHILD = """
import ctypes, sys
sys.path.insert(0, {pkg!r})
import sph_b200 as S
lib = S.load()
cfg = S.tgv_baseline_config(16)
cfg.h, cfg.kernel_scale = float({h!r}), float({scale!r})
cnt = ctypes.c_longlong(0)
fake = ctypes.c_void_p(256)
print(lib.sph_find_particle_pair_noalloc(ctypes.byref(cfg), 16, fake, fake, 0, None, None, None, None,
                                         ctypes.byref(cnt), None))
"""


@pytest.fixture(scope="module")
def built():
    import build_lib as pkg_build
    pkg_build.build()


@pytest.mark.parametrize("h,scale", [("inf", "2.0"), ("0.1", "inf"), ("1e308", "3.0")])
def test_infinite_support_is_refused(built, h, scale):
    import os
    src = CHILD.format(pkg=os.path.dirname(os.path.abspath(S.__file__)), h=h, scale=scale)
    out = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, timeout=60)
    assert out.stdout.split()[-1:] == ["-7"], out.stdout + out.stderr       # SPH_E_CONFIG
