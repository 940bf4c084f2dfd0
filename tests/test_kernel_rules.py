"""Rules that the kernels keep, read off their sources.

Every device-side wait has a limit.  A named hardware barrier has none, so no kernel whose warps can give up one by
one may use it: in the encode kernel a warp that gave up and went on arriving could fill a phase of the barrier
without the warp that waits at it, which then never came back.  What happens on the device when a wait runs
out: ``test_gpu_failure.py``.

A kernel that starts while the one before it is still at work does not read what that one writes by non-coherent
loads, which are for memory that nobody writes while the kernel runs."""
import re
import subprocess
from pathlib import Path

import pytest

from tirocinio_triennale_b200 import _build

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


def test_sums_ask_for_rate_bytes_of_several_streams_at_once():
    """Nothing stands between the loads of one stream and those of the next: added up where it is asked for, every further
    stream is one more trip to memory before the first payload."""
    kernel = _code("hc_decode.cu").split("hc_decode_kernel(", 1)[1].split("__global__", 1)[0]
    assert kernel.count("rates16(p.seg[") == 3 and not re.search(r"payload_len16\(\s*rates16\(", kernel)


def test_compute_warps_of_the_collective_kernel_leave_together():
    """They meet at hardware barriers, so a wait that ran out in one of them is no reason to go before all know: lanes
    agree within the warp, the warp tells the others at a barrier that it comes to itself."""
    code = _code("hc_kernels.cu")
    wait = code.split("bool wait_or_flag(", 1)[1].split("\n}", 1)[0]
    assert "__all_sync" in wait
    loop = code.split("int32_t d[32];", 1)[1].split("write_payload(", 1)[0]
    # the ways out of the tile loop: told and through the barrier, or told by it
    told = re.findall(r"kLeaveTotal;\s*compute_barrier\(\);\s*break;", loop)
    tellers = re.findall(r"if \(tot >= kLeaveTotal\) break;", loop)
    streams = re.findall(r"if \(W == 64\) \{\s*leave = true;\s*break;", loop)  # out of the loop over the streams
    assert (len(told), len(tellers), len(streams)) == (1, 1, 1) and loop.count("break;") == 3


@pytest.mark.parametrize("name", sorted(p.name for p in CUDA.glob("hc_*.cu*")))
def test_no_non_coherent_loads(name):
    code = _code(name)
    assert "__ldg(" not in code and ".global.nc" not in code
    # nor where the compiler may choose them: const __restrict__ arguments, in a kernel that is launched overlapped
    overlapped = re.findall(r"launch_overlapped\(dev::(\w+)", code)
    for kernel in overlapped:
        assert "__restrict__" not in code.split(kernel + "(", 1)[1].split("{", 1)[0]


def _launched_overlapped(code, headers=""):
    """{kernel: its arguments} of all kernels that a source may launch overlapped.  A launch that gets its kernel by a variable may mean
    any kernel of the source and of the headers."""
    kernels = {re.search(r"(hc_\w+)\(", k)[1]: k.split("{", 1)[0].split("hc_", 1)[1] for k in (code + headers).split("__global__")[1:]}
    names = re.findall(r"launch_overlapped\((?:dev::)?(\w+)", code)
    return kernels if any(n not in kernels for n in names) else {n: kernels[n] for n in names}


@pytest.mark.parametrize("name,headers,count", [("hc_encode.cu", [], 1), ("hc_decode.cu", ["hc_decode_step.cuh"], 3), ("hc_kernels.cu", [], 1)])
def test_every_kernel_launched_overlapped_is_looked_at(name, headers, count):
    code, headers = _code(name), "".join(_code(h) for h in headers)
    kernels = _launched_overlapped(code, headers)
    assert len(kernels) == count
    for arguments in kernels.values():
        assert "__restrict__" not in arguments
    # an argument that breaks the rule is seen, however the launch names its kernel
    for kernel in kernels:
        broken = (code + headers).replace(kernel + "(const __grid_constant__", kernel + "(const int* __restrict__ x, const __grid_constant__", 1)
        assert broken != code + headers and "__restrict__" in _launched_overlapped(broken)[kernel]


def test_no_other_source_launches_overlapped():
    names = [p.name for p in sorted(CUDA.glob("hc_*.cu*")) if p.name != "hc_host.cuh" and "launch_overlapped(" in _code(p.name)]
    assert names == ["hc_decode.cu", "hc_encode.cu", "hc_kernels.cu"]


@pytest.mark.parametrize("name,index,issued", [("hc_encode.cu", 0, "jobs"), ("hc_decode.cu", 0, "jobs"), ("hc_decode.cu", 1, "issued")])
def test_a_warp_that_gives_up_waits_for_its_copies(name, index, issued):
    """Bulk copies land in shared memory; the CTA does not leave it while one may be on its way."""
    kernels = _code(name).split("__global__")[1:]
    assert len(kernels) == {"hc_encode.cu": 1, "hc_decode.cu": 2}[name]
    kernel = kernels[index].split("\n}\n", 1)[0]
    after_the_loop = kernel.rsplit("HC_PH_COUNT();", 1)[1]
    assert re.search(r"for \(;[^;]*< %s; [^)]*\)\s*mbar_wait_bounded\(" % issued, after_the_loop)


def test_decode_of_collective_steps_keeps_the_same_rules():
    """It is launched overlapped too, through hc_decode.cu."""
    code = _code("hc_decode_step.cuh")
    assert not re.search(r'"(\\n|\\t|\s)*(bar|barrier)\.', code) and "__restrict__" not in code
    after_the_loop = code.rsplit("HC_PH_COUNT();", 1)[1]
    assert re.search(r"for \(; v < jobs; [^)]*\)\s*mbar_wait_bounded\(", after_the_loop)


@pytest.mark.skipif(_build.nvcc_path() is None, reason="needs nvcc")
@pytest.mark.parametrize("name", ["hc_encode.cu", "hc_decode.cu"])
def test_no_spills(name, tmp_path):
    """As the assembler reports them.  The add of int32 deltas (operation 2) is left out: it keeps 12 bytes there and is
    slower in the form that needs none."""
    flags = [f for f in _build.NVCC_FLAGS if f != "-lineinfo"]
    out = subprocess.run([_build.nvcc_path(), *flags, "-Xptxas", "-v", "-I", str(CUDA.parent / "include"), "-cubin",
                          str(CUDA / name), "-o", str(tmp_path / "cubin")], capture_output=True, text=True, check=True).stderr
    entries = [e for e in out.split("Compiling entry function ")[1:] if "hc_encode_solo_kernelILi2E" not in e]
    assert len(entries) >= 6
    for e in entries:
        name = e.split("'")[1]
        assert re.findall(r"(\d+) bytes spill stores, (\d+) bytes spill loads", e.split("Function properties for " + name)[1])[0] == (
            "0", "0"), name
