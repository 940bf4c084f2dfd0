"""Every device-side wait has a limit.  A named hardware barrier has none, so no kernel whose warps can give up one by
one may use it: in the encode kernel a warp that gave up and went on arriving could fill a phase of the barrier
without the warp that waits at it, which then never came back.  Read off the sources; what happens on the device
when a wait runs out: ``test_gpu_failure.py``."""
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
