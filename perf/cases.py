"""Performance cases: the work a program gives this library, through its public calls.

listed() is a spread over the calls' real range; draw(rng) gives more cases of
the same ranges.  A case is a dict of plain values:

  op       "compress", "decompress" or "batch" (many inputs in one call)
  data     where the input bytes come from (source() below)
  size     input bytes (decompress: bytes of the decoded output)
  level    1..9, the stream's header digit (and, for batch, the block size)
  block    raw bytes per block, or -1 for bzip2 1.0.8's own block format
  where    "host": ordinary host memory in, bytes out; "pinned": page-locked
           host memory in and out; "device": input in device memory (the
           stream goes to page-locked memory, decoded bytes to device memory)
  table    table selector: "plain" (the default form) or "learned"
  count, most  batch: number of inputs and the largest one's bytes

Sizes, levels and sources are those of bzip2gpu_b200.workloads (the small
Markov stream, the stress segments, the many-inputs batch, the large stream)
and of the tests.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bzip2gpu_b200 as B
import bzip2gpu_b200.selector as S
import bzip2gpu_b200.workloads as W

KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30


def _case(name, op, size, data="segments", level=9, block=900000, where="host", table="plain",
          count=0, most=0):
    return {"name": name, "op": op, "size": size, "data": data, "level": level, "block": block,
            "where": where, "table": table, "count": count, "most": most}


def listed():
    return [
        # a small message or log record: the call's own latency
        _case("compress_2KB", "compress", 2039, "markov"),
        # one full block, the library's unit of work
        _case("compress_one_block", "compress", 900000, "markov"),
        # a small file (the small Markov stream: five blocks)
        _case("compress_4MiB", "compress", 4 * MIB, "markov"),
        # bzip2's own format at a middle level, a ragged size, a changing source
        _case("compress_bzip2_format_48MB", "compress", 48_000_011, "segments", level=5, block=-1,
              where="pinned"),
        # inputs that are hard on the sort: zeros, a short period, noise, text-like
        _case("compress_stress_64MiB", "compress", 64 * MIB, "stress", where="device"),
        # the learned table selector
        _case("compress_learned_128MiB", "compress", 128 * MIB, "segments", where="device",
              table="learned"),
        # a file read into page-locked memory, end to end
        _case("compress_pinned_256MiB", "compress", 256 * MIB + 12345, "segments", where="pinned"),
        # a large stream resident on the device: the throughput form
        _case("compress_device_1GiB", "compress", GIB, "segments", where="device"),
        # many inputs of mixed size and level in one call
        _case("batch_128_inputs", "batch", 0, "segments", where="device", count=128, most=8 * MIB),
        # decoding one block: latency
        _case("decompress_one_block", "decompress", 900000, "markov"),
        # decoding a file in page-locked memory
        _case("decompress_pinned_48MB", "decompress", 48_000_011, "segments", where="pinned"),
        # decoding a large stream on the device
        _case("decompress_device_512MiB", "decompress", 512 * MIB, "segments", where="device"),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.random()
    level = rng.randint(1, 9)
    if kind < 0.15:
        return {k: v for k, v in _case("", "batch", 0, level=level, where="device",
                                       count=_log(rng, 8, 192),
                                       most=_log(rng, 64 * KIB, 4 * MIB)).items() if k != "name"}
    where = rng.choice(["host", "pinned", "device"])
    if kind < 0.45:
        size = _log(rng, KIB, 8 * MIB if where == "host" else 512 * MIB)
        c = _case("", "decompress", size, rng.choice(["markov", "segments", "stress"])
                  if size <= 64 * MIB else "segments", level=level, where=where)
    else:
        data = rng.choice(["markov", "segments", "segments", "stress"])
        hi = 8 * MIB if where == "host" else 48 * MIB if data != "segments" else 768 * MIB
        size = _log(rng, KIB, hi)
        block = rng.choice([900000, 900000, 900000, 100000 * level, -1])
        table = "learned" if data == "segments" and rng.random() < 0.2 else "plain"
        c = _case("", "compress", size, data, level, block, where, table)
    c.pop("name")
    return c


def source(data: str, n: int, seed: int):
    """n seeded bytes in device memory.

    markov    one order-1 Markov source over printable symbols with 2 % runs
    segments  the large stream: a new alphabet and skew every 64 MiB, from the
              nearly constant to the nearly uniform
    stress    quarters: zeros, a repeated 17-byte string, uniform bytes, markov
    """
    if data == "markov":
        return W.small_markov(n, seed=0xB2C0 + 7919 * seed, device=True)
    if data == "segments":
        return W.large_stream(n, seed=0xB2C4 + 7919 * seed, device=True)
    q = n // 4
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    out[q:2 * q] = torch.from_numpy(W.periodic17(q, seed=0xB2C1B + 7919 * seed)).cuda()
    if q:
        B.gen_uniform(q, 0xB2C1C + 7919 * seed, out=out[2 * q:3 * q])
    if n > 3 * q:
        B.gen_markov(n - 3 * q, 0xB2C1D + 7919 * seed, W.PRINTABLE, 0.3, 0.02, 4, 300,
                     out=out[3 * q:])
    return out


def _pinned(n):
    return torch.zeros(n, dtype=torch.uint8, pin_memory=True)


def prepare(case, seed):
    """The inputs, and the buffers a program that calls again and again keeps."""
    if case["op"] == "batch":
        # the case fixes the inputs' sizes, levels and sources; the seed their bytes
        specs = W.batch_specs(case["count"], max_size=case["most"])
        for sp in specs:
            sp.segment.seed += (7919 * seed) << 32
        total = sum(sp.size for sp in specs)
        return {"case": case, "inputs": [sp.make(device=True) for sp in specs],
                "levels": [sp.level for sp in specs],
                "out": _pinned(total + total // 16 + 4096 * len(specs))}
    n = case["size"]
    d = source(case["data"], n, seed)
    room = n + n // 32 + 65536
    if case["op"] == "decompress":
        B.set_selector("plain")
        comp = _pinned(room)
        comp = comp[:B.compress_device_into(d, comp, case["level"], case["block"])]
        if case["where"] == "device":
            return {"case": case, "in": comp.cuda(), "out": torch.empty_like(d)}
        if case["where"] == "pinned":
            src = _pinned(comp.numel())
            src.copy_(comp)
            return {"case": case, "in": src, "out": _pinned(n)}
        return {"case": case, "in": comp.numpy().tobytes(), "out": None}
    if case["table"] == "learned":
        B.selector_load(S.load())
    if case["where"] == "device":
        return {"case": case, "in": d, "out": _pinned(room)}
    if case["where"] == "pinned":
        src = _pinned(n)
        src.copy_(d)
        torch.cuda.synchronize()
        return {"case": case, "in": src, "out": _pinned(room)}
    return {"case": case, "in": d.cpu().numpy().tobytes(), "out": np.zeros(room, np.uint8)}


def run(state):
    """One call.  Streams come back in a buffer with room to spare (its rest
    stays zero) and their lengths, so that outputs have one shape for a case."""
    case = state["case"]
    src, out = state.get("in"), state["out"]
    if case["op"] == "batch":
        streams = B.compress_batch(state["inputs"], state["levels"], out=out, on_device=True)
        lengths = [len(s) for s in streams]
        return {"streams": out, "lengths": np.array(lengths, np.int64)}
    if case["op"] == "decompress":
        if case["where"] == "host":
            return np.frombuffer(B.decompress(src), np.uint8)
        return {"bytes": out, "length": B.decompress_into(src, out)}
    B.set_selector(case["table"])
    if case["where"] == "host":
        stream = B.compress(src, case["level"], case["block"])
        out[:len(stream)] = np.frombuffer(stream, np.uint8)
        return {"stream": out, "length": len(stream)}
    into = B.compress_device_into if case["where"] == "device" else B.compress_into
    return {"stream": out, "length": into(src, out, case["level"], case["block"])}


def work(case):
    """Input bytes read once and output bytes written once, at the sources'
    usual compression; flops only for the learned selector's network
    (266 kFLOP per 50-symbol group, about 0.27 symbols per input byte)."""
    n = case["size"]
    if case["op"] == "batch":
        # sizes are log-uniform from 1 KiB to `most`
        n = case["count"] * (case["most"] - KIB) / math.log(case["most"] / KIB)
    flops = 0.27 * n / 50 * 266e3 if case["table"] == "learned" else 0.0
    return {"bytes": 1.2 * n, "flops": flops}


def exact(case, seed):
    """Outputs are bytes: there is nothing to round."""
    return None
