"""Copies between the handle and the caller's arrays when something fails (a copy, an
allocation, a thread): an error code, never an abort, and nothing left in flight at the
caller's memory.  host_copy.cuh runs over a stand-in for the CUDA runtime
(host_copy_fake.cpp), so no GPU is needed."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_copy") / "fake")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-isystem", "/usr/local/cuda/include", "-o", exe,
                    os.path.join(HERE, "host_copy_fake.cpp")], check=True)
    return exe


def test_failures_leave_nothing_in_flight(program):
    out = subprocess.run([program], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout[-2000:] + out.stderr[-2000:]


def test_device_arrays_are_left_to_the_runtime(program):
    """A caller's array in device memory is copied by the runtime, never by the CPU."""
    out = subprocess.run([program, "device"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout[-2000:], out.stderr[-2000:])


def test_what_a_new_handle_takes(program):
    """A small owner locks a little ordinary memory, others take one block and the helper
    threads' block with the first large copy, an owner of large states takes both at
    once; all copies right."""
    out = subprocess.run([program, "reserve"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout[-2000:], out.stderr[-2000:])
