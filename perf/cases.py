"""The work that users of this framework have it do, as cases that can be timed.

A case is one pass of a monitoring or serving program through the public classes: clear a
sketch, insert a key stream, query it (the reference's own benchmark loop), in the sizes and
key distributions of the repository's benchmark and tests and in odd sizes between them.
Sketches are made with their default settings.

Keys are uint32 held in int32 tensors.  Skewed streams follow a bounded power law of
exponent s over `ranks` distinct keys, ranks mapped to keys by a bijection of the 32-bit
integers; everything is drawn from the seed on the device.
"""
import math

import numpy as np
import torch

DEV = "cuda"
U32 = 0xffffffff


def listed():
    return [
        # a control-plane check: a few hundred keys through a small sketch, all launch latency
        {"name": "tiny", "kind": "msws", "n": 1000, "dist": "power", "s": 1.2, "ranks": 300, "n_low": 2039,
         "n_high": 512, "query": "ranks"},
        # a serving process answers a small odd-sized batch of lookups from a warm 64 MB sketch
        {"name": "lookup_small", "kind": "lookup", "n": 1 << 23, "dist": "power", "s": 1.1, "ranks": 1 << 22,
         "n_low": 2097143, "n_high": 1 << 17, "queries": 10007},
        # one ordinary, ragged batch of moderately skewed keys into a 16 MB sketch
        {"name": "ragged_1m", "kind": "msws", "n": 1000003, "dist": "power", "s": 0.9, "ranks": 200003,
         "n_low": 524287, "n_high": 32768, "query": "ranks"},
        # the benchmark's uniform workload: 2^24 uniform keys, 8 MB low table, every key queried
        {"name": "uniform_16m", "kind": "msws", "n": 1 << 24, "dist": "uniform", "s": 0.0, "ranks": 0,
         "n_low": 262139, "n_high": 1 << 16, "query": "keys"},
        # the benchmark's default workload: 2^27 Zipf-skewed keys, 64 MB + 16 MB, distinct keys queried
        {"name": "zipf_128m", "kind": "msws", "n": 1 << 27, "dist": "power", "s": 1.1, "ranks": 1 << 24,
         "n_low": 2097143, "n_high": 1 << 17, "query": "ranks"},
        # the benchmark's mixed workload in steady alternation: batches of 2^20 operations, 90 %
        # inserts then 10 % queries, on a 256 MB table that does not fit the L2
        {"name": "mixed_hbm", "kind": "mixed", "batch": 1 << 20, "batches": 64, "dist": "power", "s": 0.8,
         "ranks": 1 << 26, "n_low": 8388593, "n_high": 1 << 19},
        # the benchmark's batched workload: 512 uneven streams, a sketch each, inserted and queried
        {"name": "batched_512", "kind": "batch", "streams": 512, "min_len": 1 << 10, "max_len": 1 << 22,
         "ranks": 1 << 20, "min_bytes": 32 << 10, "max_bytes": 16 << 20, "graph": False},
        # serving the same kind of batch at low latency: 512 short slices, recorded as a graph
        {"name": "batched_serving", "kind": "batch", "streams": 512, "min_len": 700, "max_len": 1300,
         "ranks": 1 << 20, "min_bytes": 32 << 10, "max_bytes": 1 << 20, "graph": True},
        # the plain count-min baseline at the uniform workload's bytes
        {"name": "count_min_16m", "kind": "cm", "n": 1 << 24, "dist": "uniform", "s": 0.0, "ranks": 0,
         "width": 524287, "rows": 3},
        # a sliding window: two periods inserted, the older one removed again, the newer one queried
        {"name": "window_remove", "kind": "window", "n": 3000017, "dist": "power", "s": 1.0, "ranks": 1 << 20,
         "n_low": 524287, "n_high": 1 << 16},
        # the learned split after its warm-up: routed inserts and queries of structured keys, 64 MB
        {"name": "learned_routed", "kind": "learned", "n": 1 << 24, "warmup": 1 << 22, "budget": 64 << 20,
         "slots": 1 << 17, "queries": 1 << 20},
        # a program that keeps its keys in pinned host memory and calls the host-buffer entry points
        {"name": "host_stream", "kind": "host", "n": 1 << 24, "dist": "power", "s": 1.1, "ranks": 1 << 21,
         "n_low": 524287, "n_high": 1 << 15, "query": "ranks"},
    ]


PRIMES = [2039, 4093, 8191, 16381, 32749, 65521, 131071, 262139, 524287, 1048573, 2097143, 4194301]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def keys(n):
        uniform = rng.random() < 0.3
        return {"dist": "uniform" if uniform else "power", "s": 0.0 if uniform else round(rng.uniform(0.6, 1.4), 3),
                "ranks": 0 if uniform else log_int(200, 1 << 24)}

    kind = rng.choice(["msws", "msws", "msws", "msws", "lookup", "mixed", "batch", "batch", "cm", "bucket", "window",
                       "learned", "host"])
    if kind == "mixed":
        return {"kind": kind, "batch": log_int(1 << 17, 1 << 21), "batches": rng.randint(8, 32), "dist": "power",
                "s": round(rng.uniform(0.6, 1.1), 3), "ranks": log_int(1 << 22, 1 << 26), "n_low": 8388593,
                "n_high": 1 << 19}
    if kind == "batch":
        graph = rng.random() < 0.4
        longest = log_int(500, 4000) if graph else log_int(1 << 15, 1 << 21)
        return {"kind": kind, "streams": log_int(16, 512), "min_len": max(1, longest // 64), "max_len": longest,
                "ranks": log_int(1 << 12, 1 << 20), "min_bytes": 32 << 10,
                "max_bytes": log_int(1 << 19, (1 << 20) if graph else (16 << 20)), "graph": graph}
    if kind == "learned":
        return {"kind": kind, "n": log_int(1 << 21, 1 << 25), "warmup": 1 << 22, "budget": log_int(16 << 20, 96 << 20),
                "slots": 1 << rng.randint(15, 17), "queries": log_int(1 << 16, 1 << 22)}
    if kind in ("cm", "bucket"):
        n = log_int(1 << 12, 1 << 24)
        c = {"kind": kind, "n": n, **keys(n), "width": rng.choice(PRIMES[2:9])}
        return {**c, "rows": rng.randint(1, 5)} if kind == "cm" else {**c, "m": rng.choice([8, 16, 32])}
    if kind == "window":
        n = log_int(1 << 14, 1 << 21)
    elif kind == "host":
        n = log_int(1 << 14, 1 << 24)
    elif kind == "lookup":
        n = log_int(1 << 18, 1 << 23)
    else:
        n = log_int(500, 1 << 26)
    n |= rng.randint(0, 1)
    c = {"kind": kind, "n": n, **keys(n), "n_low": rng.choice(PRIMES), "n_high": 0}
    c["n_high"] = max(64, c["n_low"] // rng.choice([1, 4, 16]))
    if kind == "lookup":
        c["queries"] = log_int(100, 1 << 22)
    elif kind == "window":
        c["s"] = min(c["s"], 1.0)
    else:
        c["query"] = "ranks" if c["ranks"] else "keys"
    return c


# ---- key streams ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _to_keys(r, salt):
    """Ranks (int64) to distinct uint32 keys: a bijection of the 32-bit integers."""
    k = (r * 0x9E3779B1 + salt) & U32
    k = k ^ (k >> 15)
    k = (k * 0x2C1B3C6D) & U32
    k = k ^ (k >> 13)
    return torch.where(k > 0x7fffffff, k - (1 << 32), k).to(torch.int32)


def _power_ranks(u, s, ranks):
    """Ranks of a bounded power law by inversion of its continuous distribution; s and ranks may
    be tensors."""
    if isinstance(s, float):
        x = torch.exp(u * math.log(ranks + 1)) if abs(s - 1) < 1e-9 else \
            (u * ((ranks + 1.0) ** (1 - s) - 1) + 1) ** (1 / (1 - s))
    else:
        x = (u * ((ranks + 1.0) ** (1 - s) - 1) + 1) ** (1 / (1 - s))
    return (x.to(torch.int64) - 1).clamp_(0, ranks - 1)


def _stream(c, n, g, salt):
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    step = 1 << 24
    for a in range(0, n, step):
        b = min(n, a + step)
        if c["dist"] == "uniform":
            out[a:b] = torch.randint(-(1 << 31), 1 << 31, (b - a,), generator=g, device=DEV, dtype=torch.int64).to(
                torch.int32)
        else:
            u = torch.rand(b - a, generator=g, device=DEV, dtype=torch.float64)
            out[a:b] = _to_keys(_power_ranks(u, float(c["s"]), c["ranks"]), salt)
    return out


def _salt(seed):
    return (seed * 0x5851F42D + 0x1405) & U32


def _inputs(c, seed):
    """Inserted keys and queried keys of the single-sketch kinds."""
    g, salt = _gen(seed), _salt(seed)
    if c["kind"] == "lookup":
        k = _stream(c, c["n"], g, salt)
        return k, _stream(c, c["queries"], g, salt)
    if c["kind"] == "window":
        return _stream(c, c["n"], g, salt), _stream(c, c["n"], g, salt)
    if c["kind"] == "mixed":
        return _stream(c, c["batch"] * c["batches"], g, salt), None
    k = _stream(c, c["n"], g, salt)
    if c.get("query", "keys") == "keys":
        return k, k
    return k, _to_keys(torch.arange(c["ranks"], device=DEV, dtype=torch.int64), salt)


def _class_keys(n, g, salt):
    u = torch.rand(2, n, generator=g, device=DEV, dtype=torch.float64)
    cls = _power_ranks(u[0], 1.0, 1 << 16)
    suf = _power_ranks(u[1], 1.2, 1 << 16)
    cls = ((cls * 0x6487 + salt) & 0xffff)
    suf = ((suf * 0x9E35 + cls * 0x3D4D) & 0xffff)
    k = (cls << 16) | suf
    return torch.where(k > 0x7fffffff, k - (1 << 32), k).to(torch.int32)


def _uneven(c, seed):
    """Lengths, exponents and sketch sizes of a batch (the case's own), the flat keys and their
    offsets."""
    from qsketch_b200 import find_greatest_prime
    rng = np.random.default_rng(c["streams"])
    n_s = c["streams"]
    lengths = np.exp(rng.uniform(np.log(c["min_len"]), np.log(c["max_len"]), n_s)).astype(np.int64)
    expo = rng.uniform(0.6, 1.4, n_s)
    nbytes = np.exp(rng.uniform(np.log(c["min_bytes"]), np.log(c["max_bytes"]), n_s)).astype(np.int64)
    n_low = np.array([find_greatest_prime(int(b) // 32) for b in nbytes], np.uint64)
    n_high = np.maximum(2, nbytes // 4 // 128).astype(np.uint64)
    off = np.zeros(n_s + 1, np.int64)
    off[1:] = np.cumsum(lengths)
    g = _gen(seed)
    offsets = torch.from_numpy(off).to(DEV)
    keys = torch.empty(int(off[-1]), dtype=torch.int32, device=DEV)
    salts = torch.randint(0, 1 << 32, (n_s,), generator=g, device=DEV, dtype=torch.int64)
    s_dev = torch.from_numpy(expo).to(DEV)
    step = 1 << 24
    for a in range(0, keys.numel(), step):
        b = min(keys.numel(), a + step)
        sid = torch.searchsorted(offsets, torch.arange(a, b, device=DEV), right=True) - 1
        u = torch.rand(b - a, generator=g, device=DEV, dtype=torch.float64)
        keys[a:b] = _to_keys(_power_ranks(u, s_dev[sid], c["ranks"]), salts[sid])
    return keys, offsets, n_low, n_high


def _cm_seeds(rows):
    return [(0x9E3779B1 * (2 * j + 1) + 0x7F4A7C14 * j) & U32 | 1 for j in range(rows)]


def _bucket_masks(m, count=1021):
    """Three distinct counters of m per mask."""
    r = np.random.default_rng(m)
    bits = np.argsort(r.random((count, m)), axis=1)[:, :3]
    return (1 << bits.astype(np.uint64)).sum(1).astype({8: np.uint8, 16: np.uint16, 32: np.uint32}[m])


# ---- what a program keeps, and one pass ------------------------------------------------------


def prepare(case, seed):
    import qsketch_b200 as qs
    c, kind = case, case["kind"]
    st = {"kind": kind}
    if kind == "batch":
        from qsketch_b200.batch import BatchedSketches
        keys, offsets, n_low, n_high = _uneven(c, seed)
        st.update(sk=BatchedSketches(n_low, n_high), keys=keys, offsets=offsets, total=keys.numel(),
                  out=torch.empty_like(keys), graph=c["graph"])
        return st
    if kind == "learned":
        from qsketch_b200.learned import LearnedSketch
        g, salt = _gen(seed), _salt(seed)
        sk = LearnedSketch(budget_bytes=c["budget"], warmup_keys=c["warmup"], table_slots=c["slots"])
        sk.insert(_class_keys(c["warmup"], g, salt))  # trains and fills the exact table
        keys = _class_keys(c["n"], g, salt)
        q = keys[:c["queries"]].clone() if c["queries"] < c["n"] else keys
        st.update(sk=sk, keys=keys, queries=q, out=torch.empty_like(q))
        return st
    keys, queries = _inputs(c, seed)
    if kind == "cm":
        sk = qs.Sketch_GPU_Thread(c["width"], c["rows"], seeds=_cm_seeds(c["rows"]))
    elif kind == "bucket":
        sk = qs.Sketch_GPU_Warp(c["width"], c["m"], hash_seed=2654435769, mask_table=_bucket_masks(c["m"]))
    else:
        sk = qs.Sketch_GPU_Sub_Warp_Level(c["n_low"], 8, c["n_high"], 32, hash_seed=2654435769)
    st["sk"] = sk
    if kind == "mixed":
        ins = c["batch"] * 9 // 10
        parts = keys.split(c["batch"])
        st["steps"] = [(p[:ins], p[ins:]) for p in parts]
        st["outs"] = [torch.empty_like(q) for _, q in st["steps"]]
        return st
    if kind == "lookup":
        sk.insert(keys)
        st.update(queries=queries, out=torch.empty_like(queries))
        return st
    if kind == "host":
        st["keys"] = keys.cpu().pin_memory()
        st["queries"] = queries.cpu().pin_memory()
        st["out"] = torch.empty_like(st["queries"]).pin_memory()
        return st
    st.update(keys=keys, queries=queries, out=torch.empty_like(queries))
    return st


def run(st):
    sk, kind = st["sk"], st["kind"]
    if kind == "lookup":
        return sk.search(st["queries"], counts=st["out"])
    if kind == "learned":
        sk.insert(st["keys"])
        return sk.search(st["queries"], counts=st["out"])
    sk.clear()
    if kind == "batch":
        if st["graph"]:
            sk.insert_graph(st["keys"], st["offsets"])
            return sk.search_graph(st["keys"], st["offsets"], st["out"])
        sk.insert(st["keys"], st["offsets"], total=st["total"])
        return sk.search(st["keys"], st["offsets"], total=st["total"], counts=st["out"])
    if kind == "mixed":
        for (ins, q), out in zip(st["steps"], st["outs"]):
            sk.insert(ins)
            sk.search(q, counts=out)
        return st["outs"]
    if kind == "host":
        sk.insert_host(st["keys"])
        return sk.search_host(st["queries"], st["out"])
    sk.insert(st["keys"])
    if kind == "window":
        sk.insert(st["queries"])
        sk.remove(st["keys"])
    return sk.search(st["queries"], counts=st["out"])


def work(case):
    """Keys read once, estimates written once, and the sketch's tables written once where a pass
    starts from a cleared sketch."""
    c, kind = case, case["kind"]
    if kind == "batch":
        n = c["streams"] * (c["max_len"] - c["min_len"]) / math.log(c["max_len"] / c["min_len"]) \
            if c["max_len"] > c["min_len"] else c["streams"] * c["max_len"]
        tables = c["streams"] * (c["max_bytes"] - c["min_bytes"]) / math.log(c["max_bytes"] / c["min_bytes"])
        return {"bytes": 12 * n + 1.2 * tables, "flops": 0}
    if kind == "learned":
        return {"bytes": 4 * c["n"] + 8 * min(c["n"], c["queries"]), "flops": 0}
    if kind == "lookup":
        return {"bytes": 8 * c["queries"], "flops": 0}
    tables = 4 * c["width"] * c["rows"] if kind == "cm" else 4 * c["width"] * c["m"] if kind == "bucket" \
        else 32 * c["n_low"] + 128 * c["n_high"]
    if kind == "mixed":
        n = c["batch"] * c["batches"]
        return {"bytes": 4 * n + 0.4 * n + tables, "flops": 0}
    if kind == "window":
        return {"bytes": 12 * c["n"] + 8 * c["n"] + tables, "flops": 0}
    q = c["ranks"] if c.get("query") == "ranks" else c["n"]
    return {"bytes": 4 * c["n"] + 8 * q + tables, "flops": 0}


# ---- the estimates in 64-bit integers --------------------------------------------------------


def _u(k):
    return k.to(torch.int64) & U32


def _min_rows(cells, table):
    return table[cells].min(dim=1).values.to(torch.int32)


def exact(case, seed):
    """Estimates of the sketches whose counters only ever add up, from plain bincounts.  The
    two-level sketches' integer state follows from the array order of their keys and has no value
    but the one the path defines."""
    c, kind = case, case["kind"]
    if kind not in ("cm", "bucket"):
        return None
    keys, queries = _inputs(c, seed)
    k, q = _u(keys), _u(queries)
    if kind == "cm":
        def cells(x):
            return torch.stack([((x * s) & U32) % c["width"] + j * c["width"]
                                for j, s in enumerate(_cm_seeds(c["rows"]))], 1)
        size = c["width"] * c["rows"]
    else:
        masks = _bucket_masks(c["m"]).astype(np.int64)
        bits = torch.tensor([[i for i in range(c["m"]) if (int(w) >> i) & 1] for w in masks], device=DEV)

        def cells(x):
            hv = (x * 2654435769) & U32
            return (hv % c["width"])[:, None] * c["m"] + bits[hv % len(masks)]
        size = c["width"] * c["m"]
    table = torch.zeros(size, dtype=torch.int64, device=DEV)
    for a in range(0, k.numel(), 1 << 22):
        table += torch.bincount(cells(k[a:a + (1 << 22)]).reshape(-1), minlength=size)
    return torch.cat([_min_rows(cells(q[a:a + (1 << 22)]), table) for a in range(0, q.numel(), 1 << 22)])
