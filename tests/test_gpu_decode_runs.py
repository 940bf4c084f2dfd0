"""Decode of stand-alone streams: payloads staged as a sequence of bytes through a ring, runs and pools, and the exchange of
totals whose words outlive a launch."""
import numpy as np
import pytest
import torch

from tirocinio_triennale_b200 import ops

pytestmark = pytest.mark.gpu
EB = 0.5  # quantised values are the values themselves


def _values(n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "wide":  # 31 planes: the longest payloads, none of whose sub-tiles ends where a staged piece does
        x = rng.integers(-2 ** 29, 2 ** 29, n)
    elif kind == "mixed":  # from no payload to the longest, block by block
        bits = np.repeat(rng.integers(0, 30, (n + 31) // 32), 32)[:n]
        x = rng.integers(-2 ** 29, 2 ** 29, n) >> (29 - bits)
    else:
        x = rng.integers(-300, 300, n)
    return x.astype(np.float32)


def _on_gpu(stream, shift):
    t = torch.zeros(stream.size + 64, dtype=torch.uint8, device="cuda")
    t[shift:shift + stream.size] = torch.from_numpy(stream)
    return t[shift:shift + stream.size]


@pytest.mark.parametrize("mode", ["outlier", "plain", "vec"])
@pytest.mark.parametrize("kind,n", [("wide", 5_000_003), ("mixed", 3_333_333), ("narrow", 148 * 20 * 1024 * 4), ("mixed", 33 * 1024 * 4 + 1)])
def test_payloads_of_all_lengths(kind, n, mode):
    x = _values(n, kind, n)
    ref = ops.cpu_compress(x, EB, mode)
    want = ops.cpu_decompress(ref, n, EB, mode)
    c = ops.Codec(n)
    got = [c.decompress(_on_gpu(ref, shift), n, EB, mode, stream_bytes=ref.size) for shift in (0, 1, 15)]
    for g in got:
        np.testing.assert_array_equal(g.cpu().numpy(), want)
    assert c.status() == 0


def test_runs_of_more_than_32_sub_tiles():
    n, eb = 148 * 20 * 1024 * 34 + 5, 1e-3
    x = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    c = ops.Codec(n)
    s, size = c.compress(x, eb)
    y = c.decompress(s, n, eb, stream_bytes=int(size))
    t = x * (torch.tensor(0.5) / torch.tensor(eb)).item()
    q = (t + 0.5).trunc() - (t < -0.5).float()
    assert torch.equal(y, q * np.float32(eb) * 2)
    assert c.status() == 0


@pytest.mark.parametrize("n,cut", [(200_000, 3), (200_000, 200_000), (6_000_000, 1), (6_000_000, 7_000_001)])
def test_stream_that_ends_early(n, cut):
    x = _values(n, "mixed", 5)
    ref = ops.cpu_compress(x, EB)
    want = ops.cpu_decompress(ref, n, EB)
    c = ops.Codec(n)
    got = c.decompress(_on_gpu(ref, 0), n, EB, stream_bytes=ref.size - cut).cpu().numpy()
    assert c.status() == 2
    rates = ref[:(n + 31) // 32].astype(np.int64)
    planes = rates & 31
    lens = np.where(rates & 128, 5 + 4 * planes + (rates >> 5 & 3), np.where(planes, 4 + 4 * planes, 0))
    lens = np.append(lens, np.zeros(-lens.size % 32, np.int64)).reshape(-1, 32).sum(1)
    there = (n + 32767) // 32768 * 1024 + np.cumsum(lens) <= ref.size - cut  # sub-tiles whose payload is complete
    mask = np.repeat(there | (lens == 0), 1024)[:n]
    np.testing.assert_array_equal(got, np.where(mask, want, 0))


@pytest.mark.parametrize("k", [1, 2, 4, 5, 8])
def test_sums_by_length_of_the_runs(k):
    sizes = (1, 1024 * 4 * 148, 1024 * 16 * 148 + 1, 1024 * 16 * 148 * 4, 1024 * 16 * 148 * 4 + 1024)
    c = ops.Codec(k * ((max(sizes) + 32767) // 32768 * 32768))
    for n in sizes:
        refs = [ops.cpu_compress(_values(n, "narrow", n + i), EB) for i in range(k)]
        got = c.decompress_sum([_on_gpu(r, i) for i, r in enumerate(refs)], n, EB, stream_bytes=[r.size for r in refs])
        want = refs[0]
        for r in refs[1:]:
            want = ops.cpu_hom_add_streams(want, r, n)
        np.testing.assert_array_equal(got.cpu().numpy(), ops.cpu_decompress(want, n, EB))
    assert c.status() == 0


@pytest.mark.parametrize("k,subs", [(3, 17), (5, 5), (5, 33), (8, 18)])
def test_sums_over_long_runs(k, subs):
    """Rate bytes are added up 16 sub-tiles of four streams at a time; every stream has payloads of its own lengths."""
    n = 148 * 16 * 1024 * subs + 1025  # some warps have a sub-tile more
    g = torch.Generator("cuda").manual_seed(k)
    c = ops.Codec(k * ((n + 32767) // 32768 * 32768))
    want, streams, sizes = torch.zeros(n, device="cuda"), [], []
    for i in range(k):
        x = torch.randint(-(3 << i), 3 << i, (n,), device="cuda", generator=g).float()
        want += x
        s, size = c.compress(x, EB)
        streams.append(s)
        sizes.append(int(size))
    assert torch.equal(c.decompress_sum(streams, n, EB, stream_bytes=sizes), want)
    assert c.status() == 0


@pytest.mark.parametrize("k,bits", [(2, 22), (3, 21), (4, 20), (5, 16), (8, 19)])
def test_sums_of_payloads_that_fill_the_ring(k, bits):
    """Four payloads of a sub-tile that fit in the ring together, that do not, and some of no bytes, by turns; the last stream ends early."""
    n = 148 * 16 * 1024 * 5 + 1025
    g = torch.Generator("cuda").manual_seed(k)
    c = ops.Codec(k * ((n + 32767) // 32768 * 32768))
    xs, streams, sizes = [], [], []
    for i in range(k):
        x = torch.randint(-2 ** bits, 2 ** bits, (n,), device="cuda", generator=g)
        less = torch.randint(0, bits + 2, (n // 1024 + 1,), device="cuda", generator=g) * (torch.arange(n // 1024 + 1, device="cuda") % 3 == 0)
        x = (x * 2 + 1 >> less.repeat_interleave(1024)[:n] + 1).float()
        s, size = c.compress(x, EB)
        xs.append(x)
        streams.append(s)
        sizes.append(int(size))
    want = sum(xs)
    assert torch.equal(c.decompress_sum(streams, n, EB, stream_bytes=sizes), want)
    assert c.status() == 0
    sizes[-1] -= 1
    want[(n - 1) // 1024 * 1024:] -= xs[-1][(n - 1) // 1024 * 1024:]
    assert torch.equal(c.decompress_sum(streams, n, EB, stream_bytes=sizes), want)
    assert c.status() == 2


@pytest.mark.parametrize("k,bits", [(2, 22), (3, 1), (4, 20), (5, 16), (8, 19)])
def test_sums_of_payloads_of_no_bytes(k, bits):
    """Sub-tiles without payload in some of the streams of a batch, and in all of them: such a copy has no bytes, such a batch no copy."""
    n = 148 * 16 * 1024 * 5 + 1025
    subs = (n + 1023) // 1024
    g = torch.Generator("cuda").manual_seed(100 + k)
    c = ops.Codec(k * ((n + 32767) // 32768 * 32768))
    in_all = torch.rand(subs, device="cuda", generator=g) < 0.2
    want, streams, sizes, empty = torch.zeros(n, device="cuda"), [], [], []
    for i in range(k):
        none = in_all | (torch.rand(subs, device="cuda", generator=g) < 0.4)
        x = torch.randint(-2 ** bits, 2 ** bits, (n,), device="cuda", generator=g)
        x = x.masked_fill(none.repeat_interleave(1024)[:n], 0).float()
        s, size = c.compress(x, EB)
        want += x
        streams.append(s)
        sizes.append(int(size))
        empty.append((s[:subs * 32].reshape(subs, 32) == 0).all(1))  # rate bytes
    empty = torch.stack(empty)
    for half in (empty[:4], empty[4:]):  # the streams of a batch
        assert len(half) == 0 or half.all(0).sum() > subs / 10
        assert len(half) < 2 or (half.any(0) & ~half.all(0)).sum() > subs / 10
    assert torch.equal(c.decompress_sum(streams, n, EB, stream_bytes=sizes), want)
    assert c.status() == 0


def test_launches_of_all_grids_behind_one_another():
    """A launch leaves words of the exchange as they are; the next one, with more CTAs or fewer, starts from there."""
    rng = np.random.default_rng(3)
    grids = [148, 1, 65, 64, 147, 14, 66, 148, 78, 79, 91, 92, 146, 2] + list(rng.integers(1, 149, 40))
    most = 148 * 4 * 1024
    c = ops.Codec(2 * (most + 32768))
    x = _values(most, "narrow", 9)
    runs = []
    for g in grids:
        n = int(g) * 4 * 1024 - int(rng.integers(0, 4096))
        ref = ops.cpu_compress(x[:n], EB)
        runs.append((n, ref, _on_gpu(ref, 0)))
    torch.cuda.synchronize()
    got = []
    for n, ref, s in runs:  # one launch right behind the other
        got.append((c.decompress(s, n, EB, stream_bytes=ref.size), c.decompress_sum([s, s], n, EB, stream_bytes=[ref.size] * 2)))
    for (n, ref, _), (one, two) in zip(runs, got):
        want = ops.cpu_decompress(ref, n, EB)
        np.testing.assert_array_equal(one.cpu().numpy(), want)
        np.testing.assert_array_equal(two.cpu().numpy(), 2 * want)
    assert c.status() == 0
