"""Stand-alone kernels at the edges of their split: sub-tiles of 1024 values, chunks of up to 15 (adds) or 23 (compress)
sub-tiles per CTA of 148, runs with and without a shared pool (decode), and blocks beyond the reach of the float form."""
import numpy as np
import pytest
import torch

from tirocinio_triennale_b200 import ops

pytestmark = pytest.mark.gpu
EB = 1e-3


def _data(n, seed):
    """Smooth values; some blocks zero, some with quantised values around 2^20, 2^23, 2^24 and 2^26, some of them jumping."""
    rng = np.random.default_rng(seed)
    x = np.cumsum(rng.standard_normal(n, dtype=np.float32) * np.float32(4e-3), dtype=np.float32)
    x -= np.repeat(x[::1024], 1024)[:n]
    for b in rng.choice((n + 31) // 32, size=max(1, n // 3200), replace=False):
        block = x[32 * b:32 * b + 32]
        kind = b % 6
        if kind == 0:
            block[:] = 0
        elif kind == 5:
            block[:] = rng.choice([-1, 1], block.size) * np.float32(2.0 ** 24 * EB)
        else:
            block += np.float32(2.0 ** (20, 23, 24, 26)[kind - 1] * 2 * EB)
    return x


def _gpu(x, shift=0):
    """On the device, `shift` elements behind a 16-byte boundary, with room to read a little further."""
    t = torch.zeros(x.size + 64, dtype=torch.from_numpy(x[:0]).dtype, device="cuda")
    t[shift:shift + x.size] = torch.from_numpy(x)
    return t[shift:shift + x.size]


@pytest.mark.parametrize("mode", ["outlier", "plain", "vec"])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 148 * 4 * 1024 + 1, 148 * 15 * 1024, 148 * 15 * 1024 + 1,
                               148 * 23 * 1024, 148 * 23 * 1024 + 1, 13_000_077])
def test_edges_of_the_split(n, mode):
    xs = [_data(n, s) for s in range(3)]
    shift = n & 1  # operands off the boundary go past the TMA unit
    gx = [_gpu(x, shift) for x in xs]
    c = ops.Codec(3 * ((n + 32767) // 32768 * 32768))
    ref = [ops.cpu_compress(x, EB, mode) for x in xs]
    gs = [_gpu(r, 3 * shift) for r in ref]
    sizes = [r.size for r in ref]

    def same(got, want):
        out, size = got
        assert int(size) == want.size
        np.testing.assert_array_equal(out[:want.size].cpu().numpy(), want)

    # launched behind one another, looked at afterwards
    comp = [c.compress(g, EB, mode) for g in gx]
    dec = c.decompress(gs[0], n, EB, mode, out=torch.full_like(gx[0], 7.0), stream_bytes=sizes[0])
    add = c.hom_add(gs[0], gx[1], EB, mode, stream_bytes=sizes[0])
    deltas = c.hom_add_deltas(gs[0], c.quant_pred(gx[1], EB, mode), n, mode, stream_bytes=sizes[0])
    both = c.hom_add_streams(gs[0], gs[1], n, mode, a_bytes=sizes[0], b_bytes=sizes[1])
    multi = c.hom_add_multi(gs[:2], gx[2], EB, mode, stream_bytes=sizes[:2])
    for got, want in zip(comp, ref):
        same(got, want)
    np.testing.assert_array_equal(dec.cpu().numpy(), ops.cpu_decompress(ref[0], n, EB, mode))
    two = ops.cpu_hom_add(ref[0], xs[1], EB, mode)
    for got in (add, deltas, both):
        same(got, two)
    three = ops.cpu_hom_add(two, xs[2], EB, mode)
    same(multi, three)
    if mode == "outlier":
        total = c.decompress_sum(gs, n, EB, stream_bytes=sizes)
        np.testing.assert_array_equal(total.cpu().numpy(), ops.cpu_decompress(three, n, EB))
    assert c.status() == 0


def test_batch_of_very_different_sizes_in_a_codec_for_their_sum():
    lens = [5, 3_000_001, 1024, 40_000, 148 * 4 * 1024 + 7, 31, 32769, 1]
    xs = [_data(n, 7 + i) for i, n in enumerate(lens)]
    c = ops.Codec(sum((n + 32767) // 32768 * 32768 for n in lens))
    outs, sizes = c.compress_batch([_gpu(x) for x in xs], EB)
    for out, size, x in zip(outs, sizes.tolist(), xs):
        want = ops.cpu_compress(x, EB)
        assert size == want.size
        np.testing.assert_array_equal(out[:size].cpu().numpy(), want)
    assert c.status() == 0


@pytest.mark.parametrize("mode", ["outlier", "plain", "vec"])
def test_batch_of_several_rounds(mode):
    """Payloads that wait for their place belong to any of eight arrays; some are as long as a payload gets."""
    rng = np.random.default_rng(8)
    xs = [_data(1_200_000 + 777 * i, i) for i in range(8)]
    for i in (3, 7):  # 31 planes in every block
        xs[i] = rng.integers(-2 ** 29, 2 ** 29, xs[i].size).astype(np.float32) * np.float32(2 * EB)
    c = ops.Codec(sum((x.size + 32767) // 32768 * 32768 for x in xs))
    outs, sizes = c.compress_batch([_gpu(x) for x in xs], EB, mode)
    for out, size, x in zip(outs, sizes.tolist(), xs):
        want = ops.cpu_compress(x, EB, mode)
        assert size == want.size
        np.testing.assert_array_equal(out[:size].cpu().numpy(), want)
    assert c.status() == 0


@pytest.mark.parametrize("n,shift", [(1023, 0), (4099, 1), (70_001, 3)])
def test_chain_through_one_ragged_operand(n, shift):
    """Every call reads what the call before it has just written into the same buffer, past the TMA unit (ragged, or
    off the 16-byte boundary); small enough that several of the launches are on an SM at the same time."""
    c = ops.Codec(2 * 32768 * (n // 32768 + 1))
    refs = [ops.cpu_compress(_data(n, s), EB) for s in range(24)]
    gs = [_gpu(r) for r in refs]
    x = _gpu(np.zeros(n, np.float32), shift)
    got = []
    for i, r in enumerate(refs):
        c.decompress(gs[i], n, EB, out=x, stream_bytes=r.size)
        got.append((c.compress(x, EB), c.hom_add(gs[0], x, EB, stream_bytes=refs[0].size)))
    assert c.status() == 0
    for r, ((out, size), (added, added_size)) in zip(refs, got):
        y = ops.cpu_decompress(r, n, EB)
        for o, k, want in ((out, size, ops.cpu_compress(y, EB)), (added, added_size, ops.cpu_hom_add(refs[0], y, EB))):
            assert int(k) == want.size
            np.testing.assert_array_equal(o[:want.size].cpu().numpy(), want)
