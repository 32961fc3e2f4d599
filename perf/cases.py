"""Performance cases of the block codec: what a program built on this
package has it do, from one block per call to the largest batches, through
the package's public entry points.

A case names an operation, the data it runs on and the shape of the batch:

  op      "call"       one block through PackUint32, UnpackUint32, GetUint32
          "pack"       BatchCodec.pack of a whole batch
          "unpack"     BatchCodec.unpack of a packed batch
          "roundtrip"  BatchCodec.pack, then BatchCodec.unpack of the result
          "get"        BatchCodec.get at random (stream, position) pairs
          "index"      index_stream over a packed stream without an index
  data    "uniform"    uint32 uniform in [0, 2^bits)
          "outliers"   uint32 uniform in [0, 2^8), 2% uniform in [2^8, 2^32),
                       10% of the blocks all equal
          "lists"      uint32 strictly increasing lists, gaps 1 + Geom(1/64)
          "mixed64"    uint64 streams: a third 2^40 + uniform [0, 2^20), a
                       third full range, a third random walks from 2^62
  flag    the pack flag (Delta, NoFOR, NoPatch or their sums)
  values, streams      totals of the batch; the stream lengths are
                       log-uniform, so most streams end in a partial block
"""
import math

import numpy as np
import torch

import utlpfor_b200 as U

# Packed bytes per value of each data set, measured with the CPU oracle.
_PACKED = {("outliers", 0): 1.024, ("outliers", U.NoFOR): 1.12, ("outliers", U.NoPatch): 3.42,
           ("lists", U.Delta): 1.56, ("lists", U.Delta | U.NoFOR): 1.56,
           ("mixed64", 0): 4.3, ("mixed64", U.Delta): 4.34}


def listed():
    return [
        # One block per call from the host: what a caller of the reference's
        # own API does first, and where only latency counts.
        {"name": "call_block", "op": "call", "data": "outliers", "flag": 0, "values": 128, "streams": 1},
        # A few short streams of odd lengths: a request of a serving loop.
        {"name": "few_short_streams", "op": "roundtrip", "data": "outliers", "flag": 0, "values": 5003, "streams": 9},
        # 2^20 11-bit values: the plain round trip, latency and ramp-up bound.
        {"name": "uniform_roundtrip", "op": "roundtrip", "data": "uniform", "bits": 11, "flag": 0,
         "values": 1 << 20, "streams": 1},
        # The benchmark's workload, each direction: 2^28 values with outliers.
        {"name": "outliers_pack", "op": "pack", "data": "outliers", "flag": 0, "values": 1 << 28, "streams": 1},
        {"name": "outliers_unpack", "op": "unpack", "data": "outliers", "flag": 0, "values": 1 << 28, "streams": 1},
        # The same values without patching: large blocks of 32-bit payload,
        # in ragged streams.
        {"name": "nopatch_roundtrip", "op": "roundtrip", "data": "outliers", "flag": U.NoPatch,
         "values": 30000001, "streams": 40},
        # 1000 posting lists, delta coded: an index writer, an index reader
        # that takes whole lists, and one that looks single postings up.
        {"name": "lists_pack", "op": "pack", "data": "lists", "flag": U.Delta, "values": 100000007, "streams": 1000},
        {"name": "lists_unpack", "op": "unpack", "data": "lists", "flag": U.Delta, "values": 100000007,
         "streams": 1000},
        {"name": "lists_get", "op": "get", "data": "lists", "flag": U.Delta, "values": 100000007, "streams": 1000,
         "queries": 1 << 20},
        # uint64 streams of all three shapes the codec has, each direction.
        {"name": "mixed64_pack", "op": "pack", "data": "mixed64", "flag": U.Delta, "values": 1 << 26, "streams": 512},
        {"name": "mixed64_unpack", "op": "unpack", "data": "mixed64", "flag": U.Delta, "values": 1 << 26,
         "streams": 512},
        # A stream packed elsewhere, whose block offsets have to be found.
        {"name": "index_stream", "op": "index", "data": "outliers", "flag": U.NoFOR, "values": (1 << 26) + 77,
         "streams": 1},
    ]


def draw(rng):
    data = rng.choice(["uniform", "outliers", "outliers", "lists", "lists", "mixed64"])
    op = rng.choice(["pack", "unpack", "pack", "unpack", "roundtrip", "get", "index", "call"])
    if op == "call":
        return {"op": "call", "data": "outliers", "flag": rng.choice([0, U.NoFOR, U.NoPatch]),
                "values": rng.randint(1, 128), "streams": 1}
    case = {"op": op, "data": data}
    if data == "uniform":
        case["bits"] = rng.randint(1, 31)
        case["flag"] = 0
    elif data == "outliers":
        case["flag"] = rng.choice([0, U.NoFOR, U.NoPatch])
    elif data == "lists":
        case["flag"] = rng.choice([U.Delta, U.Delta | U.NoFOR])
    else:
        case["flag"] = rng.choice([0, U.Delta])
    hi = {"mixed64": 25.5, "lists": 26.5}.get(data, 27.0)
    if op == "roundtrip":
        hi -= 1
    n = int(2 ** rng.uniform(12, hi)) | 1
    case["values"] = n
    if op == "index":
        case["streams"] = 1
        if data in ("lists", "mixed64"):
            case["data"], case["flag"] = "outliers", rng.choice([0, U.NoFOR, U.NoPatch])
    else:
        # lists stay short enough for their sums to fit 32 bits
        lo = max(1, n >> 19)
        case["streams"] = int(math.exp(rng.uniform(math.log(lo), math.log(max(lo, min(2000, n // 256)) + 1))))
    if op == "get":
        case["queries"] = int(2 ** rng.uniform(8, 20))
    return case


def _is64(case):
    return case["data"] == "mixed64"


def _val_off(case):
    """Stream table: log-uniform lengths that add up to the case's values."""
    n, k = case["values"], case["streams"]
    if k == 1:
        return np.array([0, n], dtype=np.uint64)
    rng = np.random.default_rng(n + 1000003 * k)
    w = np.exp(rng.uniform(0.0, math.log(8192.0), k))
    cut = np.floor(np.cumsum(w) * (n / w.sum())).astype(np.int64)
    cut[-1] = n
    return np.concatenate([[0], cut]).astype(np.uint64)


def _per_stream_sum(x, vo):
    """Running sums of x (int64) that start again at every stream."""
    cs = torch.cumsum(x, 0)
    lens = torch.from_numpy(np.diff(vo.astype(np.int64))).to(x.device)
    starts = torch.from_numpy(vo[:-1].astype(np.int64)).to(x.device)
    base = torch.where(starts > 0, cs[(starts - 1).clamp(min=0)], torch.zeros_like(starts))
    return cs - torch.repeat_interleave(base, lens)


def _values(case, seed, vo, device):
    n = case["values"]
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    if case["data"] == "uniform":
        return torch.randint(0, 1 << case["bits"], (n,), device=device, dtype=torch.int64, generator=gen).to(torch.int32)
    if case["data"] == "outliers":
        v = torch.randint(0, 256, (n,), device=device, dtype=torch.int32, generator=gen)
        m = torch.rand(n, device=device, generator=gen) < 0.02
        k = int(m.sum())
        v[m] = torch.randint(256, 2**32, (k,), device=device, dtype=torch.int64, generator=gen).to(torch.int32)
        vb = v[:n // 128 * 128].view(-1, 128)
        same = torch.rand(vb.shape[0], device=device, generator=gen) < 0.10
        c = torch.randint(0, 256, (vb.shape[0],), device=device, dtype=torch.int32, generator=gen)
        vb.copy_(torch.where(same[:, None], c[:, None], vb))
        return v
    if case["data"] == "lists":
        u = 1.0 - torch.rand(n, device=device, dtype=torch.float64, generator=gen)
        gaps = 1 + torch.floor(torch.log(u) / math.log(1.0 - 1.0 / 64.0)).to(torch.int64)
        return _per_stream_sum(gaps, vo).to(torch.int32)
    kind = torch.arange(case["streams"], device=device) % 3
    kind = torch.repeat_interleave(kind, torch.from_numpy(np.diff(vo.astype(np.int64))).to(device))
    v = _per_stream_sum(torch.randint(-1000, 1001, (n,), device=device, dtype=torch.int64, generator=gen), vo) + 2**62
    near = 2**40 + torch.randint(0, 2**20, (n,), device=device, dtype=torch.int64, generator=gen)
    v = torch.where(kind == 0, near, v)
    full = torch.randint(-2**63, 2**63 - 1, (n,), device=device, dtype=torch.int64, generator=gen)
    return torch.where(kind == 1, full, v)


def _queries(case, seed, vo, device):
    """Uniform streams among the non-empty ones, a uniform position in each."""
    gen = torch.Generator(device=device)
    gen.manual_seed(seed + 1)
    lens = torch.from_numpy(np.diff(vo.astype(np.int64))).to(device)
    live = torch.nonzero(lens > 0).flatten()
    q = case["queries"]
    s = live[torch.randint(0, live.numel(), (q,), device=device, generator=gen)]
    pos = (torch.rand(q, device=device, dtype=torch.float64, generator=gen) * lens[s]).to(torch.int64)
    return s.to(torch.int32), torch.minimum(pos, lens[s] - 1)


def prepare(case, seed):
    if case["op"] == "call":
        v = _values(case, seed, _val_off(case), "cpu").numpy().view(np.uint32)
        return {"op": "call", "flag": case["flag"], "values": v, "pos": int(seed) % case["values"],
                "room": U.MaxBlockLength32(case["flag"])}
    vo = _val_off(case)
    values = _values(case, seed, vo, "cuda")
    codec = U.BatchCodec(vo, flag=case["flag"], is64=_is64(case))
    codec.packed.zero_()
    state = {"op": case["op"], "codec": codec}
    if case["op"] in ("pack", "roundtrip"):
        state["values"] = values
    else:
        codec.pack(values)
    if case["op"] in ("unpack", "roundtrip"):
        state["out"] = torch.zeros_like(values)
    elif case["op"] == "get":
        state["q_stream"], state["q_pos"] = _queries(case, seed, vo, "cuda")
        state["out"] = torch.zeros(case["queries"], dtype=values.dtype, device="cuda")
        state["status"] = torch.zeros(case["queries"], dtype=torch.int32, device="cuda")
    elif case["op"] == "index":
        state["packed"] = codec.packed[:codec.packed_len].clone()
        del state["codec"]
    return state


def run(state):
    op = state["op"]
    if op == "call":
        block = bytes(U.PackUint32(state["flag"], state["values"]))
        values, consumed = U.UnpackUint32(block)
        one = U.GetUint32(state["pos"], block)
        return {"block": np.frombuffer(block.ljust(state["room"], b"\0"), dtype=np.uint8), "values": values,
                "consumed": consumed, "one": one}
    if op == "index":
        return {"block_off": U.index_stream(state["packed"])}
    codec = state["codec"]
    if op == "get":
        codec.get(state["q_stream"], state["q_pos"], state["out"], state["status"])
        return {"values": state["out"], "status": state["status"], "err": codec.err}
    if op != "unpack":
        codec.pack(state["values"])
    if op != "pack":
        codec.unpack(state["out"])
    got = {"err": codec.err}
    if op != "unpack":
        got["packed"], got["block_off"] = codec.packed, codec.block_off
    if op != "pack":
        got["values"] = state["out"]
    return got


def exact(case, seed):
    """The values an unpack or a Get gives back; packed bytes and offsets
    have no value but their own."""
    if case["op"] not in ("unpack", "get"):
        return None
    vo = _val_off(case)
    values = _values(case, seed, vo, "cuda")
    if case["op"] == "unpack":
        return {"values": values, "err": None}
    s, pos = _queries(case, seed, vo, "cuda")
    return {"values": values[torch.from_numpy(vo[:-1].astype(np.int64)).cuda()[s.long()] + pos], "status": None,
            "err": None}


def work(case):
    n, size = case["values"], 8 if _is64(case) else 4
    blocks = -(-n // 128)
    if case["data"] == "uniform":
        per = (case["bits"] + 3) // 4 / 2.0 + 4 / 128.0
    else:
        per = _PACKED[(case["data"], case["flag"])]
    packed = per * n
    if case["op"] == "get":
        # a query, its two table entries, a sector of its block, its answer
        return {"bytes": case["queries"] * (12 + 16 + 32 + size + 4), "flops": 0}
    if case["op"] == "index":
        return {"bytes": packed + 8 * blocks, "flops": 0}
    one = size * n + packed + 8 * blocks
    if case["op"] == "call":
        return {"bytes": 2 * one + packed + 4, "flops": 0}
    return {"bytes": (2 if case["op"] == "roundtrip" else 1) * one, "flops": 0}
