"""Sums of streams in bit planes against the oracle: magnitudes at the edges of the planes that the kernel keeps, sums that grow out
of them and that wrap like an int32, first values inside and outside the planes, blocks without payload among them."""
import numpy as np
import pytest
import torch

from tirocinio_triennale_b200 import ops

pytestmark = pytest.mark.gpu


def _walk(n, bits, seed):
    """Values (step size 1) whose differences inside a block are of up to `bits` bits, with first values of 0 to 24 bits."""
    rng = np.random.default_rng(seed)
    d = rng.integers(-(2 ** bits) + 1, 2 ** bits, n) if bits else np.zeros(n, np.int64)
    d = d >> rng.integers(0, bits + 1, -(-n // 32)).repeat(32)[:n]  # blocks of fewer planes, and of none
    d[::32] = rng.integers(-(2 ** 24), 2 ** 24, d[::32].size) >> rng.integers(0, 26, d[::32].size)
    q = np.concatenate([np.cumsum(b) for b in np.split(d, range(32, n, 32))])
    return np.clip(q, -(2 ** 29), 2 ** 29).astype(np.float32)


def _gpu(a):
    return torch.from_numpy(np.concatenate([a, np.zeros(32, a.dtype)])).cuda()


@pytest.mark.parametrize("mode", ["outlier", "plain", "vec"])
@pytest.mark.parametrize("bits", [0, 4, 8, 9, 12, 13, 15, 16, 17, 19, 20, 24, 28])
def test_sums_of_streams(bits, mode):
    n, eb, k = 5 * 1024 + 77, 0.5, 8
    codec = ops.Codec((k + 1) * 32768)
    xs = [_walk(n, max(0, bits - (i % 3 == 1)), 100 * bits + i) for i in range(k + 1)]
    streams = [ops.cpu_compress(x, eb, mode) for x in xs]
    gpu = [_gpu(s) for s in streams]
    want = streams[0]
    for i in range(1, k):
        last, want = want, ops.cpu_hom_add_streams(want, streams[i], n, mode)
        if i in (1, 2, 6, 7):
            out, size = codec.hom_add_multi(gpu[:i + 1], torch.from_numpy(xs[k]).cuda(), eb, mode,
                                            stream_bytes=[s.size for s in streams[:i + 1]])
            np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), ops.cpu_hom_add(want, xs[k], eb, mode))
        out, size = codec.hom_add_streams(_gpu(last), gpu[i], n, mode, a_bytes=last.size, b_bytes=streams[i].size)
        np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), want)
        if mode != "vec":  # (streams with the stride-1 predictor only)
            y = codec.decompress_sum(gpu[:i + 1], n, eb, stream_bytes=[s.size for s in streams[:i + 1]])
            np.testing.assert_array_equal(y.cpu().numpy(), ops.cpu_decompress(want, n, eb, mode))
    assert codec.status() == 0


def _with_gaps(n, bits, seed):
    """Differences of up to `bits` bits, and blocks that are all zero: next to one another in the sub-tiles, in some of which all are."""
    rng = np.random.default_rng(seed)
    blocks = -(-n // 32)
    d = rng.integers(-(2 ** bits) + 1, 2 ** bits, (blocks, 32))
    d[:, 0] >>= rng.integers(0, bits + 1, blocks)
    d[rng.random(blocks) < 0.5] = 0
    d[(np.arange(blocks) // 32 + seed) % 5 == 0] = 0
    return np.clip(d.cumsum(1).reshape(-1)[:n], -(2 ** 29), 2 ** 29).astype(np.float32)


@pytest.mark.parametrize("mode", ["outlier", "plain", "vec"])
@pytest.mark.parametrize("bits", [1, 4, 8, 12, 16, 17, 18, 20, 24])
def test_sums_with_blocks_of_no_planes(bits, mode):
    """What stands where the sign map of a block without payload would be belongs to another block, and has no effect."""
    n, eb, k = 10 * 1024 + 77, 0.5, 8
    codec = ops.Codec((k + 1) * 32768)
    xs = [_with_gaps(n, bits, 10 * bits + i) for i in range(k + 1)]
    streams = [ops.cpu_compress(x, eb, mode) for x in xs]
    for s in streams:
        planes = (s[:10 * 32] & 31).reshape(10, 32)  # of whole sub-tiles
        assert ((planes == 0).any(1) & (planes.max(1) >= bits)).sum() >= 7 and (planes.max(1) == 0).sum() >= 2
    gpu = [_gpu(s) for s in streams]
    want = streams[0]
    for i in range(1, k):
        last, want = want, ops.cpu_hom_add_streams(want, streams[i], n, mode)
        out, size = codec.hom_add_streams(_gpu(last), gpu[i], n, mode, a_bytes=last.size, b_bytes=streams[i].size)
        np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), want)
        if i in (1, 2, 6, 7):
            sizes = [s.size for s in streams[:i + 1]]
            out, size = codec.hom_add_multi(gpu[:i + 1], torch.from_numpy(xs[k]).cuda(), eb, mode, stream_bytes=sizes)
            np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), ops.cpu_hom_add(want, xs[k], eb, mode))
            if mode != "vec":  # (streams with the stride-1 predictor only)
                y = codec.decompress_sum(gpu[:i + 1], n, eb, stream_bytes=sizes)
                np.testing.assert_array_equal(y.cpu().numpy(), ops.cpu_decompress(want, n, eb, mode))
    assert codec.status() == 0


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("k,bits", [(2, 6), (2, 10), (8, 8), (3, 10), (2, 11), (2, 14), (8, 12), (3, 14), (5, 14), (8, 15), (8, 16), (2, 20)])
def test_decode_of_sums_at_the_edges(k, bits, sign):
    """Every difference as large as its planes allow, all of one sign, so that the sums reach the bound that the kernel goes by; first
    values that leave what it adds up in floats, and that just do not."""
    eb = 0.5
    firsts = np.array([0, 1, -1, 2 ** 19, 2 ** 22 // k, 2 ** 22 // k - 1, -(2 ** 22) // k, -(2 ** 22) // k - 1, 2 ** 22, -(2 ** 23)])
    q = firsts.repeat(32) + sign * np.tile(np.arange(32) * (2 ** bits - 1), firsts.size)
    n = q.size
    codec = ops.Codec((k + 1) * 32768)
    stream = ops.cpu_compress(q.astype(np.float32), eb)
    want = stream
    for _ in range(k - 1):
        want = ops.cpu_hom_add_streams(want, stream, n)
    gpu = _gpu(stream)
    y = codec.decompress_sum([gpu] * k, n, eb, stream_bytes=[stream.size] * k)
    np.testing.assert_array_equal(y.cpu().numpy(), ops.cpu_decompress(want, n, eb))
    assert codec.status() == 0


def _any_stream(n, planes, first_bytes, seed):
    """A stream of random rate bytes and random payloads: outlier blocks with a |d_0| of 32 bits, and with planes that hold something
    for element 0 too, as this library does not write them."""
    rng = np.random.default_rng(seed)
    blocks = -(-n // 32)
    planes = rng.integers(0, planes + 1, blocks)
    rates = np.where(rng.random(blocks) < 0.5, planes, 128 | rng.integers(0, first_bytes, blocks) << 5 | planes)
    rates = np.append(rates, np.zeros(-blocks % 1024, rates.dtype))
    lens = np.where(rates & 128, 5 + 4 * (rates & 31) + (rates >> 5 & 3), np.where(rates & 31, 4 + 4 * (rates & 31), 0))
    return np.append(rates, rng.integers(0, 256, lens.sum())).astype(np.uint8)


@pytest.mark.parametrize("planes,first_bytes", [(0, 4), (4, 1), (8, 2), (10, 2), (12, 4), (14, 2), (16, 4), (18, 1), (31, 4)])
def test_sums_of_streams_that_another_encoder_wrote(planes, first_bytes):
    """d_0 of an outlier block is its bytes, 31 bits of them, and nothing but them."""
    n, eb, k = 37 * 1024 + 77, 0.5, 8
    codec = ops.Codec((k + 1) * 65536)
    x = _walk(n, 8, planes)
    streams = [_any_stream(n, planes, first_bytes, 10 * planes + i) for i in range(k)]
    gpu = [_gpu(s) for s in streams]
    sizes = [s.size for s in streams]
    for mode in ("outlier", "plain", "vec"):
        out, size = codec.hom_add(gpu[0], torch.from_numpy(x).cuda(), eb, mode, stream_bytes=sizes[0])
        np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), ops.cpu_hom_add(streams[0], x, eb, mode))
        out, size = codec.hom_add_streams(gpu[0], gpu[1], n, mode, a_bytes=sizes[0], b_bytes=sizes[1])
        np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), ops.cpu_hom_add_streams(streams[0], streams[1], n, mode))
    want = streams[0]
    for i in range(1, k):
        want = ops.cpu_hom_add_streams(want, streams[i], n)
        if i in (1, 2, 4, 7):
            y = codec.decompress_sum(gpu[:i + 1], n, eb, stream_bytes=sizes[:i + 1])
            np.testing.assert_array_equal(y.cpu().numpy(), ops.cpu_decompress(want, n, eb))
            out, size = codec.hom_add_multi(gpu[:i + 1], torch.from_numpy(x).cuda(), eb, stream_bytes=sizes[:i + 1])
            np.testing.assert_array_equal(out[:int(size)].cpu().numpy(), ops.cpu_hom_add(want, x, eb))
    assert codec.status() == 0
