"""Clearing a status zeroes the whole workspace; the host waits for it, because the handle's next call may come on a
stream that does not order itself behind the default one and would lose its exchange words in mid-launch.  The same
goes for the zeroing of a new workspace.  Runs the library's host code on a stand-in for the CUDA runtime."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from tirocinio_triennale_b200 import _build

CALLS = """
import ctypes as C, sys
lib = C.CDLL(sys.argv[1])
pending, allocation = C.CDLL(None).fake_pending, C.CDLL(None).fake_allocation
allocation.restype = C.c_void_p
def word(p, i, v):
    C.cast(p, C.POINTER(C.c_uint32))[i] = v
vp, out = C.c_void_p, C.c_void_p()
def handle(create, *args):
    assert create(C.byref(out), *args) == 0
    assert pending() == 0, "zeroing of a new workspace"
handle(lib.hc_codec_create, C.c_size_t(1 << 20))
word(allocation(0), 2, 3)  # its workspace
assert lib.hc_codec_status(out, 0) == 3 and lib.hc_codec_status(out, 1) == 3
assert pending() == 0, "hc_codec_status"
assert lib.hc_codec_status(out, 1) == 0

region = C.create_string_buffer(1 << 20)
base = (vp * 1)(C.addressof(region) + 255 & ~255)
handle(lib.hc_comm_create, 0, 1, C.c_size_t(4096), base, None)
word(allocation(1), 34, 6)  # workspace, then size words
assert lib.hc_comm_status(out, 1) == 6
assert pending() == 0, "hc_comm_status"
assert lib.hc_comm_status(out, 1) == 0

scratch = vp()
C.CDLL(None).cudaGetSymbolAddress(C.byref(scratch), None)
word(scratch, 2, 1)
assert lib.hc_noalloc_status(0) == 1 and lib.hc_noalloc_status(1) == 1
assert pending() == 0, "hc_noalloc_status"
assert lib.hc_noalloc_status(0) == 0

print("done")
"""


@pytest.mark.skipif(_build.nvcc_path() is None and not (_build.LIBDIR / "libhomcomp_b200.so").exists(),
                    reason="needs the built library")
def test_host_waits_for_the_clearing(tmp_path):
    fake = tmp_path / "libfake_runtime.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", str(Path(__file__).with_name("fake_runtime.cpp")), "-o", str(fake)],
                   check=True)
    r = subprocess.run([sys.executable, "-c", CALLS, str(_build.build_cuda())], capture_output=True, text=True,
                       timeout=120, env={**os.environ, "LD_PRELOAD": str(fake)})
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stdout + r.stderr
