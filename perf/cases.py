"""Workloads by which changes to this framework's speed are judged.

``listed()`` gives named cases, ``draw(rng)`` further ones of the same ranges.
``prepare`` builds what a program holds before the call (keys on the GPU, a
filter, output buffers), ``run`` makes one pass through the public batch API and
returns its results, ``work`` the bytes that pass cannot do without.

Kinds of work:

* ``fill``    clear a filter and insert one batch up to ``load`` (insertManySorted
              when ``sorted``, else insertMany), then look up a sample;
* ``step``    the benchmark's step: fill, a half-positive lookup batch, deletes;
* ``lookup``  containsMany of ``n`` keys, half of them stored;
* ``churn``   a filter at ``load``: delete ``n`` stored keys, look some keys up, insert the deleted ones again;
* ``stream``  clear a filter and fill it by ``batches`` equal insertMany calls;
* ``set``     a filter set: every filter's batch inserted in one call, then as
              many lookups in another.

Results are membership flags and occupancy counts.  They do not depend on the
order in which concurrent inserts land: a lookup's answer is fixed by which
(bucket pair, tag) entries are stored, not by where in the pair they sit.
"""
import math

import numpy as np
import torch

import __graft_entry__

cfb = __graft_entry__.package()

GOLDEN = 0x9E3779B97F4A7C15


def _case(name, kind, slots, load, **more):
    c = {"name": name, "kind": kind, "slots": slots, "load": load, "bits": 16, "key_bytes": 8, "evict": "BFS",
         "alt": "xor", "n": 0, "batches": 0, "sorted": False, "results": False}
    c.update(more)
    return c


def listed():
    return [
        # One request of a service that asks a filter synchronously: launch and wait dominate.
        _case("lookup_request", "lookup", 1 << 20, 0.95, n=1000),
        # A small expiring window: a few thousand entries leave and come back, per-key results asked for.
        _case("churn_request", "churn", 1 << 20, 0.9, n=4097, results=True),
        # The benchmark's small configuration, rebuilt in one insertMany.
        _case("fill_small", "fill", 1 << 20, 0.95),
        # A join: the probe side, 4-byte keys, is many times the build side that the filter holds.
        _case("lookup_join", "lookup", 1 << 22, 0.95, key_bytes=4, n=20_000_001),
        # A set of uneven filters (per tenant or per shard of a store), built and asked in one call each.
        _case("set_step", "set", 1 << 16, 0.9, n=512),
        # k-mers streamed into a compact 8-bit filter by batches below one key per bucket.
        _case("stream_8bit", "stream", 1 << 26, 0.95, bits=8, batches=20),
        # 32-bit tags, DFS eviction, which keys were stored reported back.
        _case("fill_32bit_results", "fill", 1 << 26, 0.9, bits=32, evict="DFS", sorted=True, results=True),
        # A capacity that is no power of two under the Offset policy, part-filled by insertMany.
        _case("fill_offset", "fill", 100_000_000, 0.8, alt="offset", evict="DFS"),
        # The benchmark's medium configuration.
        _case("fill_medium", "fill", 1 << 28, 0.95, sorted=True),
        # Lookups in a table far beyond L2.
        _case("lookup_large", "lookup", 1 << 30, 0.95, n=100_000_007),
        # A large window at high load: expire a batch, insert it again.
        _case("churn_large", "churn", 1 << 30, 0.95, n=20_000_003),
        # The benchmark's step on its large configuration.
        _case("step_large", "step", 1 << 31, 0.95, sorted=True),
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["fill", "fill", "lookup", "lookup", "churn", "stream", "set"])
    c = {"kind": kind, "bits": rng.choice([16, 16, 8, 32]), "key_bytes": rng.choice([8, 8, 4]),
         "evict": rng.choice(["BFS", "DFS"]), "alt": "xor", "n": 0, "batches": 0, "sorted": rng.random() < 0.5,
         "results": rng.random() < 0.3, "load": round(rng.uniform(0.3, 0.95), 3)}
    slots = _log_int(rng, 1 << 14, 1 << 29)
    if kind == "set":
        c.update(bits=rng.choice([16, 8]), key_bytes=8, slots=_log_int(rng, 1 << 12, 1 << 18),
                 n=_log_int(rng, 16, 1024))
        return c
    if c["bits"] == 16 and rng.random() < 0.3:
        c["alt"] = rng.choice(["addsub", "offset"])
    else:
        slots = 1 << (slots.bit_length() - 1)  # the table is a power of two: so is the capacity asked for
    c["slots"] = slots
    if kind == "lookup":
        c["n"] = _log_int(rng, 500, 1 << 26)
    elif kind == "churn":
        c["n"] = max(1, min(_log_int(rng, 500, 1 << 24), int(slots * c["load"]) // 2))
    elif kind == "stream":
        c["slots"] = slots = min(slots, 1 << 27)
        c["batches"] = rng.randint(2, 24)
    return c


# ------------------------------------------------------------------- inputs

def _mix(x):
    """splitmix64's finaliser on int64 tensors (arithmetic wraps modulo 2^64)."""
    def lsr(z, s):
        return (z >> s) & ((1 << (64 - s)) - 1)

    z = (x ^ lsr(x, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ lsr(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ lsr(z, 31)


def _keys(seed, n, key_bytes, chunk=1 << 26):
    """splitmix64 outputs of `seed` as `n` 8-byte keys (their low halves as 4-byte keys) on the GPU."""
    out = torch.empty(n, dtype=torch.int64 if key_bytes == 8 else torch.int32, device="cuda")
    step = GOLDEN - (1 << 64)
    for a in range(0, n, chunk):
        m = min(chunk, n - a)
        first = (int(seed) * 0x632BE59BD9B4E019 + (a + 1) * GOLDEN) % (1 << 64)
        x = torch.arange(m, dtype=torch.int64, device="cuda") * step
        out[a:a + m] = _mix(x + (first - (1 << 64) if first >= 1 << 63 else first))
    return out


def _queries(stored, seed, n, key_bytes):
    """`n` keys in random order, about half of them among `stored`."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    q = _keys(2 * seed + (1 << 40), n, key_bytes)
    chunk = 1 << 26
    for a in range(0, n, chunk):
        m = min(chunk, n - a)
        at = torch.randint(stored.numel(), (m,), device="cuda", generator=g)
        q[a:a + m] = torch.where((at & 1) == 0, stored[at], q[a:a + m])
    return q


def _config(case):
    bits = case["bits"]
    return cfb.CuckooConfig(
        T="uint64_t" if case["key_bytes"] == 8 else "uint32_t", bitsPerTag=bits, maxEvictions=500, blockSize=256,
        bucketSize=8 if bits == 32 else 16, AltBucketPolicy=case["alt"],
        evictionPolicy=cfb.EvictionPolicy[case["evict"]])


def _sample(n):
    """Lookups made after a fill of n keys."""
    return min(n, max(1 << 16, n // 32))


def _flags(n):
    return torch.zeros(n, dtype=torch.bool, device="cuda")


def _prepare_set(case, seed):
    nf, top = case["n"], case["slots"]
    rng = np.random.default_rng(nf)  # the filters' sizes are the case's, the keys the seed's
    caps = np.exp(rng.uniform(np.log(top / 64), np.log(top * 16), nf)).astype(np.int64) + 16
    sizes = np.minimum(rng.lognormal(np.log(top / 3), 1.5, nf), case["load"] * caps).astype(np.int64)
    offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)).cuda()
    n = int(offsets[-1])
    keys = _keys(2 * seed + 1, n, 8)
    # every other lookup asks for the key inserted at the same place of the same filter's batch
    probes = torch.where(torch.arange(n, device="cuda") % 2 == 0, keys, _keys(2 * seed + (1 << 40), n, 8))
    return {"set": cfb.CuckooFilterSet(_config(case), caps), "keys": keys, "probes": probes, "offsets": offsets,
            "filters": torch.arange(nf, dtype=torch.int32, device="cuda"), "stored": _flags(n), "found": _flags(n)}


def _fill(f, s):
    insert = f.insertManySorted if s["sorted"] else f.insertMany
    return insert(s["keys"], d_output=s["stored"])


def prepare(case, seed):
    if case["kind"] == "set":
        return {"kind": "set", **_prepare_set(case, seed)}
    f = cfb.CuckooFilter(_config(case), case["slots"])
    n = int(case["load"] * case["slots"])
    keys = _keys(2 * seed + 1, n, case["key_bytes"])
    s = {"kind": case["kind"], "filter": f, "keys": keys, "sorted": case["sorted"],
         "stored": _flags(n) if case["results"] and case["kind"] == "fill" else None}
    kind = case["kind"]
    if kind == "step":
        q = n // 8
        s.update(queries=_queries(keys, seed, q, case["key_bytes"]), found=_flags(q),
                 gone=keys[:n // 32].clone(), removed=_flags(n // 32))
    elif kind == "fill":
        q = _sample(n)
        s.update(queries=_queries(keys, seed, q, case["key_bytes"]), found=_flags(q))
    elif kind == "stream":
        q = _sample(n)
        s.update(queries=_queries(keys, seed, q, case["key_bytes"]), found=_flags(q),
                 parts=list(torch.tensor_split(keys, case["batches"])))
    elif kind == "lookup":
        f.insertManySorted(keys)
        s.update(queries=_queries(keys, seed, case["n"], case["key_bytes"]), found=_flags(case["n"]))
        del s["keys"]
    else:
        f.insertManySorted(keys)
        m = case["n"]
        q = m // 4 + 1
        s.update(keys=keys[:m].clone(), removed=_flags(m), stored=_flags(m) if case["results"] else None,
                 queries=_queries(keys, seed, q, case["key_bytes"]), found=_flags(q))
    return s


def run(s):
    kind = s["kind"]
    if kind == "set":
        fs = s["set"]
        fs.clear()
        fs.insert_async(s["keys"], s["offsets"], s["filters"], s["stored"])
        fs.contains_async(s["probes"], s["offsets"], s["filters"], s["found"])
        fs.sync()
        return {"stored": s["stored"], "found": s["found"]}
    f = s["filter"]
    if kind == "lookup":
        return {"found": f.containsMany(s["queries"], s["found"])}
    if kind == "churn":
        low = f.deleteMany(s["keys"], s["removed"])
        f.containsMany(s["queries"], s["found"])
        high = f.insertMany(s["keys"], d_output=s["stored"])
        return {"removed": s["removed"], "found": s["found"], "stored": s["stored"], "low": low, "high": high}
    f.clear()
    if kind == "stream":
        occupied = [f.insertMany(part) for part in s["parts"]]
        return {"occupied": occupied, "found": f.containsMany(s["queries"], s["found"])}
    out = {"occupied": _fill(f, s), "stored": s["stored"], "found": f.containsMany(s["queries"], s["found"])}
    if kind == "step":
        out["left"] = f.deleteMany(s["gone"], s["removed"])
        out["removed"] = s["removed"]
    return out


def work(case):
    """Bytes: keys read, flags written, and the buckets that a pass has to touch (at most the table, once
    read and once written where it changes).  A stored key needs one bucket, an absent one two."""
    kind = case["kind"]
    kb, slot = case["key_bytes"], case["bits"] // 8
    bucket = slot * (8 if case["bits"] == 32 else 16)
    if kind == "set":
        per = min(case["slots"] / 3, case["load"] * case["slots"]) * case["n"]
        return {"bytes": per * (2 * (kb + 1) + 2 * slot), "flops": 0}
    table = case["slots"] * slot
    n = int(case["load"] * case["slots"])
    if kind == "lookup":
        return {"bytes": case["n"] * (kb + 1) + min(table, 1.5 * case["n"] * bucket), "flops": 0}
    if kind == "churn":
        m, q = case["n"], case["n"] // 4 + 1
        return {"bytes": m * (2 * kb + 1 + (1 if case["results"] else 0)) + 4 * min(table, m * bucket)
                + q * (kb + 1) + min(table, 1.5 * q * bucket), "flops": 0}
    total = n * kb + table + (n if case["results"] else 0)  # the table is written once: it starts empty
    q = n // 8 if kind == "step" else _sample(n)
    total += q * (kb + 1) + min(table, 1.5 * q * bucket)
    if kind == "stream":
        total += (case["batches"] - 1) * 2 * min(table, n / max(1, case["batches"]) * bucket)
    if kind == "step":
        total += n // 32 * (kb + 1) + 2 * min(table, n // 32 * bucket)
    return {"bytes": total, "flops": 0}
