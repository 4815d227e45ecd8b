"""Every entry point that works on the GPU makes the handle's device current first: a
host thread starts on device 0, wherever the handle lives, and a kernel or a clear
issued to another device's stream fails.  Read from the source, as one GPU shows no
difference."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "sph-2d_b200", "csrc", "sph_b200.cu")

# no GPU work: host fields only, or a constant
HOST_ONLY = {"sph_set_body_motion", "sph_set_time", "sph_restart_size"}
# sph_init creates the handle on the current device; sph_free sets it in destroy()
OTHER = {"sph_init", "sph_free"}


def test_entry_points_set_their_device():
    src = open(SRC).read()
    src = src[src.index('extern "C" {'):]
    bodies = re.findall(r"^(?:int|size_t) (sph_\w+)\(.*?\) \{\n(.*?)^\}", src, flags=re.S | re.M)
    names = {n for n, _ in bodies}
    assert len(names) > 20 and HOST_ONLY | OTHER <= names
    for name, body in bodies:
        if name not in HOST_ONLY | OTHER:
            assert "cudaSetDevice(h->device)" in body, name
