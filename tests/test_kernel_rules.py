"""Rules that the kernels keep, read off their sources.

Every device-side wait has a limit.  A named hardware barrier has none, so no kernel whose warps can give up one by
one may use it: in the encode kernel a warp that gave up and went on arriving could fill a phase of the barrier
without the warp that waits at it, which then never came back.  What happens on the device when a wait runs
out: ``test_gpu_failure.py``.

A kernel that starts while the one before it is still at work does not read what that one writes by non-coherent
loads, which are for memory that nobody writes while the kernel runs."""
import re
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parent.parent / "csrc" / "cuda"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CUDA / name).read_text())


@pytest.mark.parametrize("name", ["hc_encode.cu", "hc_decode.cu", "hc_warp.cuh", "hc_block.cuh", "hc_device.cuh"])
def test_no_hardware_barrier_among_warps_that_can_leave(name):
    assert not re.search(r'"(\\n|\\t|\s)*(bar|barrier)\.', _code(name))


def test_block_wide_barriers_of_encode_stand_before_the_roles_part():
    kernel = _code("hc_encode.cu").split("hc_encode_solo_kernel(", 1)[1]
    assert "__syncthreads" in kernel.split("clerk(p, sh", 1)[0]
    assert "__syncthreads" not in kernel.split("clerk(p, sh", 1)[1]


@pytest.mark.parametrize("name", sorted(p.name for p in CUDA.glob("hc_*.cu*")))
def test_no_non_coherent_loads(name):
    code = _code(name)
    assert "__ldg(" not in code and ".global.nc" not in code
    # nor where the compiler may choose them: const __restrict__ arguments, in a kernel that is launched overlapped
    overlapped = re.findall(r"launch_overlapped\(dev::(\w+)", code)
    for kernel in overlapped:
        assert "__restrict__" not in code.split(kernel + "(", 1)[1].split("{", 1)[0]
