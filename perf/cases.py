"""The work that users of this library have it do, as measurable cases.

A case is a dict of plain values: ``op`` names the public entry point, the other keys its sizes and
options.  Everything goes through ``ops.Codec`` (the device codec on torch tensors) and
``parallel.CompressedAllreduce`` (the collective; with one rank it compresses and decodes the buffer).
Data sets, error bounds and sizes are those of this repository's benchmark, sweeps and trainer.

  compress          fp32 -> stream: the first half of every use of the codec
  decompress        stream -> fp32: the other half
  hom_add           stream (+) fp32 -> stream: one hop of a ring, accumulation of gradients in
                    compressed form
  hom_add_streams   stream (+) stream -> stream: combining two stored or received contributions
  reduce            several streams (+) fp32 -> stream -> fp32: the reduce step of an allreduce over
                    k + 1 ranks, and the decode of its result
  sum               several streams -> fp32: the receiving half of the one-step allreduce
  batch             the gradients of one transformer block, compressed by one launch, stream lengths
                    read and the streams put behind one another in one message
  allreduce         the collective on device buffers
  allreduce_host    the collective on pinned host buffers, the host waiting for the result
"""
import math
import os

import torch
import torch.distributed as dist

from tirocinio_triennale_b200 import ops
from tirocinio_triennale_b200.parallel import CompressedAllreduce
from tirocinio_triennale_b200.utils import datagen

LARGEST = 1 << 26  # values: the 512 x 512 x 256 field, 256 MB


def listed():
    return [
        # a small message of the sweep (4 KB): nothing but fixed costs
        {"name": "compress_4KB", "op": "compress", "n": 1024, "data": "sinusoid", "eb": 1e-3, "mode": "outlier"},
        # a layer-sized tensor with a ragged tail
        {"name": "decompress_400KB_ragged", "op": "decompress", "n": 100_003, "data": "gradient", "eb": 1e-4,
         "mode": "outlier"},
        # the smooth 3-D field, loose and tight error bound: the largest single arrays
        {"name": "compress_field_256MB", "op": "compress", "n": LARGEST, "data": "blob", "eb": 1e-3, "mode": "outlier"},
        {"name": "decompress_field_256MB", "op": "decompress", "n": LARGEST, "data": "blob", "eb": 1e-5,
         "mode": "outlier"},
        # the stride-4 predictor on normal-distributed values at the reference's test error bound
        {"name": "compress_vec_40MB", "op": "compress", "n": 10_000_000, "data": "normal", "eb": 1e-4, "mode": "vec"},
        # one hop of a ring over gradient-like values, not a whole number of blocks
        {"name": "hom_add_64MB_ragged", "op": "hom_add", "n": (1 << 24) - 5, "data": "gradient", "eb": 1e-4,
         "mode": "outlier"},
        # two stored contributions in the plain layout; random walk: values far outside the step size
        {"name": "hom_add_streams_16MB", "op": "hom_add_streams", "n": 1 << 22, "data": "randomwalk", "eb": 1e-4,
         "mode": "plain"},
        # the reduce step at 8 ranks and 64 MB per rank
        {"name": "reduce_7_streams_8MB", "op": "reduce", "n": 1 << 21, "k": 7, "data": "gradient", "eb": 1e-4},
        # the receiving half of the one-step allreduce at 4 ranks and 4 MB
        {"name": "sum_4_streams_4MB", "op": "sum", "n": 1 << 20, "k": 4, "data": "gradient", "eb": 1e-4},
        # gradients of one block of the trainer's model
        {"name": "batch_block_768", "op": "batch", "width": 768, "data": "gradient", "eb": 1e-5, "mode": "outlier"},
        # the headline benchmark on one GPU, device buffers and host buffers
        {"name": "allreduce_64MB", "op": "allreduce", "n": 1 << 24, "data": "gradient", "eb": 1e-4},
        {"name": "allreduce_host_64MB", "op": "allreduce_host", "n": 1 << 24, "data": "gradient", "eb": 1e-4},
    ]


# (data set, error bounds it is used with)
DATA = [("gradient", (1e-4, 1e-5)), ("sinusoid", (1e-3, 1e-5)), ("blob", (1e-3, 1e-5)), ("normal", (1e-4, 1e-3)),
        ("randomwalk", (1e-4, 1e-3))]
# how many values an op takes at most, so that no drawn case costs more than the largest listed one
MOST = {"compress": LARGEST, "decompress": LARGEST, "hom_add": LARGEST // 2, "hom_add_streams": LARGEST // 2,
        "reduce": LARGEST // 2, "sum": LARGEST // 2, "allreduce": LARGEST // 4, "allreduce_host": LARGEST // 4}


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    op = rng.choice(["compress", "compress", "decompress", "decompress", "hom_add", "hom_add", "hom_add_streams",
                     "reduce", "sum", "batch", "allreduce", "allreduce_host"])
    data, bounds = rng.choice(DATA)
    case = {"op": op, "data": data, "eb": rng.choice(bounds)}
    if op == "batch":
        case.update(width=_log_uniform(rng, 64, 1536), data="gradient", eb=rng.choice((1e-4, 1e-5)))
    elif op in ("reduce", "sum"):
        case["k"] = rng.randint(1 if op == "reduce" else 2, 7)
        case["n"] = _log_uniform(rng, 1024, MOST[op] // (case["k"] + 1))
    else:
        case["n"] = _log_uniform(rng, 1024, MOST[op])
    if op in ("compress", "decompress", "hom_add", "hom_add_streams", "batch"):
        case["mode"] = rng.choice(["outlier", "outlier", "outlier", "outlier", "plain", "vec"])
    return case


def _lengths(case):
    """Values of every array of the case; weights and biases of one transformer block for ``batch``."""
    if case["op"] != "batch":
        return [case["n"]]
    d = case["width"]
    return [3 * d * d, 3 * d, d * d, d, 4 * d * d, 4 * d, 4 * d * d, d]


def _values(case, n, seed, device="cuda"):
    data = case["data"]
    if data == "gradient":
        return datagen.gradient_like(n, seed, device)
    if data == "sinusoid":
        return datagen.sinusoid_field(n, seed, device)
    if data == "blob":
        nz = -(-n // (512 * 256))
        return datagen.blob_field_3d((nz, 512, 256), seed, device)[:n].clone()
    if data == "normal":
        return datagen.from_distribution(n, "normal", seed, device)
    # random walk with unit steps, summed as whole numbers so that the same seed gives the same values
    steps = datagen.from_distribution(n, "normal", seed, device)
    return ((steps * 1024).round().long().cumsum(0).double() / 1024).float()


def _stream(codec, x, case):
    """``x`` compressed: (buffer, length)."""
    buf, size = codec.compress(x, case["eb"], case.get("mode", "outlier"))
    return buf.clone(), int(size.item())


def _comm(n):
    if not dist.is_initialized():
        os.environ.setdefault("GLOO_SOCKET_IFNAME", "lo")
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    return CompressedAllreduce(n)


def prepare(case, seed):
    op, eb, mode = case["op"], case["eb"], case.get("mode", "outlier")
    seed = 16 * seed
    lens = _lengths(case)
    n = lens[0]
    s = {"op": op, "eb": eb, "mode": mode, "n": n}
    if op == "batch":
        s["codec"] = ops.Codec(len(lens) * (-(-max(lens) // 32768) * 32768))
        s["xs"] = [_values(case, m, seed + i) for i, m in enumerate(lens)]
        s["message"] = torch.zeros(sum(ops.max_compressed_bytes(m) for m in lens), dtype=torch.uint8, device="cuda")
        return s
    if op in ("allreduce", "allreduce_host"):
        s["comm"] = _comm(n)
        s["send"] = _values(case, n, seed)
        s["recv"] = torch.zeros(n, device="cuda")
        if op == "allreduce_host":
            s["send"], s["recv"] = s["send"].cpu().pin_memory(), s["recv"].cpu().pin_memory()
        return s
    k = case.get("k", 2 if op == "hom_add_streams" else 0 if op == "compress" else 1)
    s["codec"] = codec = ops.Codec((k + 1) * (-(-n // 32768) * 32768))  # room for k input streams
    pairs = [_stream(codec, _values(case, n, seed + 1 + i), case) for i in range(k)]
    s["streams"], s["bytes"] = [p[0] for p in pairs], [p[1] for p in pairs]
    if op in ("compress", "hom_add", "reduce"):
        s["x"] = _values(case, n, seed)
    if op in ("compress", "hom_add", "hom_add_streams"):  # the buffers that the program sends from
        s["out"] = torch.zeros(ops.max_compressed_bytes(n) + 16, dtype=torch.uint8, device="cuda")
        s["size"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    else:
        s["y"] = torch.zeros(n, device="cuda")
    return s


def run(s):
    op, eb, mode, n = s["op"], s["eb"], s["mode"], s["n"]
    if op == "compress":
        return s["codec"].compress(s["x"], eb, mode, out=s["out"], size=s["size"])
    if op == "decompress":
        return s["codec"].decompress(s["streams"][0], n, eb, mode, out=s["y"], stream_bytes=s["bytes"][0])
    if op == "hom_add":
        return s["codec"].hom_add(s["streams"][0], s["x"], eb, mode, out=s["out"], size=s["size"],
                                  stream_bytes=s["bytes"][0])
    if op == "hom_add_streams":
        a, b = s["streams"]
        return s["codec"].hom_add_streams(a, b, n, mode, out=s["out"], size=s["size"], a_bytes=s["bytes"][0],
                                          b_bytes=s["bytes"][1])
    if op == "reduce":
        stream, size = s["codec"].hom_add_multi(s["streams"], s["x"], eb, stream_bytes=s["bytes"])
        return s["codec"].decompress(stream, n, eb, out=s["y"]), size
    if op == "sum":
        return s["codec"].decompress_sum(s["streams"], n, eb, out=s["y"], stream_bytes=s["bytes"])
    if op == "batch":
        outs, sizes = s["codec"].compress_batch(s["xs"], eb, mode)
        at = 0
        for o, m in zip(outs, sizes.tolist()):
            s["message"][at:at + m].copy_(o[:m])
            at += m
        return s["message"], sizes
    if op == "allreduce":
        return s["comm"].allreduce(s["send"], s["recv"], eb)
    out = s["comm"].allreduce_host(s["send"], s["recv"], eb)
    torch.cuda.current_stream().synchronize()  # the caller uses the result on the host
    return out


def _stream_bytes(case, n):
    """Length of the stream of n values of the case, from a sample of at most 1 Mi values."""
    m = min(n, 1 << 20)
    x = _values(case, m, 1, "cpu").numpy()
    return ops.cpu_compress(x, case["eb"], case.get("mode", "outlier")).size * (n / m)


def work(case):
    """Inputs read once, outputs written once; on host buffers that is what crosses PCIe."""
    op, lens = case["op"], _lengths(case)
    n = sum(lens)
    raw = 4.0 * n
    if op in ("allreduce", "allreduce_host"):
        # one rank: the values come back quantised.  The stream between the two halves never has to be stored.
        return {"bytes": 2 * raw, "flops": 0.0}
    coded = sum(_stream_bytes(case, m) for m in lens)
    k = case.get("k", 1)
    moved = {"compress": raw + coded, "batch": raw + coded, "decompress": coded + raw, "hom_add": raw + 2 * coded,
             "hom_add_streams": 3 * coded, "reduce": raw + (k + 1) * coded + raw, "sum": k * coded + raw}
    return {"bytes": moved[op], "flops": 0.0}


def tolerance(case):
    return "exact"  # integer arithmetic between one quantisation and one scaling, both with fixed rounding
