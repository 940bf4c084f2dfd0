"""The kernels of the multi-rank collectives on one GPU: every rank's region lies on it and the ranks take turns, one
launch of all of them after the other on one stream, so that every flag a kernel looks for is up before it starts.
Same host code, kernels and bits as with a GPU per rank; what is missing is two ranks' kernels at the same time."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

from datasets import gradient_like, smooth
from tirocinio_triennale_b200 import _lib, ops

pytestmark = pytest.mark.gpu
EB = 1e-4
ALGORITHM = {"ring": 0, "direct": 1, "onestep": 2}


class Ranks:
    def __init__(self, world, max_count, timeout_ms=5000):
        self.lib, self.world = _lib.cuda(), world
        nbytes = int(self.lib.hc_comm_symmetric_bytes(world, max_count))
        self.regions = [torch.zeros(nbytes + 256, dtype=torch.uint8, device="cuda") for _ in range(world)]
        bases = (C.c_void_p * world)(*[(r.data_ptr() + 255) // 256 * 256 for r in self.regions])
        torch.cuda.synchronize()
        self.comms = []
        for r in range(world):
            h = C.c_void_p()
            _lib.check(self.lib.hc_comm_create(C.byref(h), r, world, max_count, bases, None), "comm_create")
            self.comms.append(h)
        self.each("hc_comm_set_timeout_ms", timeout_ms)

    def each(self, name, *args):
        for h in self.comms:
            _lib.check(getattr(self.lib, name)(h, *args), name)

    def call(self, r, x, y, first=0, last=1 << 30):
        _lib.check(self.lib.hc_comm_set_steps(self.comms[r], first, last), "set_steps")
        _lib.check(self.lib.hc_allreduce(self.comms[r], x.data_ptr(), y.data_ptr(), x.numel(), EB,
                                         torch.cuda.current_stream().cuda_stream), "allreduce")

    def allreduce(self, xs, ys, algorithm):
        self.each("hc_comm_set_algorithm", ALGORITHM[algorithm])
        self.each("hc_comm_set_small_count", 0)
        for step in range({"ring": self.world + 1, "direct": 3, "onestep": 2}[algorithm]):
            for r in range(self.world):
                self.call(r, xs[r], ys[r], step, step + 1)

    def status(self, r):
        return self.lib.hc_comm_status(self.comms[r], 1)

    def close(self):
        torch.cuda.synchronize()
        for h in self.comms:
            self.lib.hc_comm_destroy(h)


def _inputs(world, n, shift=0):
    bufs = [(smooth if r % 2 else gradient_like)(n, seed=100 + r) for r in range(world)]
    xs = []
    for b in bufs:
        t = torch.zeros(n + 8, device="cuda")
        t[shift:shift + n] = torch.from_numpy(b)
        xs.append(t[shift:shift + n])
    return bufs, xs


# 1 value a rank and less, one tile, chunks of different rate bytes, more tiles than CTAs (compress 592, adds 444)
@pytest.mark.parametrize("world,n", [(2, 1), (2, 33), (2, 1048589), (2, 5_000_003), (3, 100_000), (4, 8193), (8, 70_001),
                                     (8, 8 * 120 * 4096 + 5)])
@pytest.mark.parametrize("algorithm", ["direct", "ring", "onestep"])
def test_forms_match_the_oracle(world, n, algorithm):
    shift = n & 1  # operands off the 16-byte boundary too
    bufs, xs = _inputs(world, n, shift)
    want = ops.cpu_ring_allreduce(bufs, EB)[0]
    ranks = Ranks(world, world * n if algorithm == "onestep" else n)
    for sparse, variant in ((1, 0), (0, 1), (1, 2)):  # tiles at fixed offsets or packed; both shapes of the add
        ranks.each("hc_comm_set_sparse_tiles", sparse)
        ranks.each("hc_comm_set_shares", 0, 0, variant)
        ys = [torch.full_like(x, -7.0) for x in xs]
        ranks.allreduce(xs, ys, algorithm)
        for r in range(world):
            assert ranks.status(r) == 0
            np.testing.assert_array_equal(ys[r].cpu().numpy(), want)
    sizes = (C.c_uint64 * 16)()
    _lib.check(ranks.lib.hc_comm_last_stream_bytes(ranks.comms[0], sizes, 16), "last_stream_bytes")
    if algorithm == "onestep":
        assert sizes[0] == ops.cpu_compress(bufs[0], EB).size
    ranks.allreduce(xs, xs, algorithm)  # in place
    for r in range(world):
        assert ranks.status(r) == 0
        np.testing.assert_array_equal(xs[r].cpu().numpy(), want)
    ranks.close()


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("algorithm", ["direct", "ring", "onestep"])
def test_a_rank_whose_peers_never_call(algorithm, variant):
    """Flags that nothing raises: the waits of every role run out, the call ends with status 6 or 3, and after a resync
    the ranks' next call is an ordinary one."""
    world, n = 4, 2_000_003
    bufs, xs = _inputs(world, n)
    ranks = Ranks(world, world * n, timeout_ms=50)
    ranks.each("hc_comm_set_algorithm", ALGORITHM[algorithm])
    ranks.each("hc_comm_set_small_count", 0)
    ranks.each("hc_comm_set_shares", 0, 0, variant)
    ranks.each("hc_comm_set_overlap", 0)  # the launches of the call one after the other
    ys = [torch.full_like(x, -7.0) for x in xs]
    for _ in range(5):
        t0 = time.time()
        ranks.call(0, xs[0], ys[0])
        torch.cuda.synchronize()
        assert time.time() - t0 < 10
        assert ranks.status(0) in (3, 6)
    numbers = (C.c_uint32 * 2)()
    _lib.check(ranks.lib.hc_comm_call_numbers(ranks.comms[0], numbers), "call_numbers")
    ranks.each("hc_comm_resync", numbers[0], numbers[1])
    ranks.each("hc_comm_set_timeout_ms", 5000)
    ranks.allreduce(xs, ys, algorithm)
    want = ops.cpu_ring_allreduce(bufs, EB)[0]
    for r in range(world):
        assert ranks.status(r) == 0
        np.testing.assert_array_equal(ys[r].cpu().numpy(), want)
    ranks.close()
