"""Which path a batch takes by itself, and the kernels behind it, against the oracle."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gpu_parity import dev, host_u8, image, make  # noqa: E402

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kb,bits,bs", [(8, 8, 8), (4, 8, 16), (8, 8, 64), (8, 16, 4), (8, 16, 16), (4, 16, 32),
                                        (8, 16, 128), (8, 32, 2), (8, 32, 8), (4, 32, 16)])
@pytest.mark.parametrize("per_bucket", [1, 40])
def test_lookups_tell_near_misses_apart(cfb, orc, kb, bits, bs, per_bucket):
    """The tag test of every width on buckets full of the query's tag +- 1 and
    with one bit flipped, of empty slots and of all ones; a few keys per bucket
    and many (40 per bucket, which used to be segment-staged)."""
    f, o = make(cfb, orc, kb, bits, bs, 0, 500, 64 * bs)
    keys = orc.splitmix64(7 + bits + bs, per_bucket * f.getNumBuckets() + 3)
    if kb == 4:
        keys = keys.astype(np.uint32)
    i1, i2, fp = (np.asarray(a) for a in o.candidates(keys))
    rng = np.random.default_rng(bits + bs + per_bucket)
    top = (1 << bits) - 1
    slots = rng.choice(np.array([0, 1, 2, top, top - 1], np.uint64), size=(f.getNumBuckets(), bs))
    for j in range(len(keys)):  # near misses of the key's tag, and the tag itself for one key in four
        t, b = int(fp[j]), int(i1[j] if j & 1 else i2[j])
        for v in (t ^ 1, t ^ (1 << (bits - 1)), (t + 1) & top, (t - 1) & top) + ((t,) if j % 4 == 0 else ()):
            slots[b, rng.integers(bs)] = v
    o.table[:] = slots.astype({8: np.uint8, 16: np.uint16, 32: np.uint32}[bits]).reshape(-1).view(np.uint8)
    f.load_table(torch.from_numpy(o.table.copy()).cuda())
    want = o.contains(keys)
    assert 0 < int(want.sum()) < len(keys) or per_bucket > 1
    d = dev(keys)
    assert np.array_equal(host_u8(f.containsMany(d)), want)
    for kpt in (1, 2, 4):
        f.setOption(cfb.OPT_LOOKUP_KPT, kpt)
        assert np.array_equal(host_u8(f.containsMany(d)), want)
    f.setOption(cfb.OPT_LOOKUP_KPT, 0)
    f.setOption(cfb.OPT_STAGING, cfb.STAGING_SEGMENT)
    assert np.array_equal(host_u8(f.containsMany(d)), want)
    assert np.array_equal(image(f), o.table)


POLICY = {"xor": "XorAltBucketPolicy", "addsub": "AddSubAltBucketPolicy", "offset": "OffsetAltBucketPolicy"}


def filled_and_emptied(cfb, f, batches, results, sorted_=False):
    """Inserts the batches, then checks the table by what it answers and by
    taking every key out again: a wrong or missing entry leaves a delete that
    fails or a slot that is not zero."""
    total = 0
    for keys in batches:
        ok = torch.zeros(keys.numel(), dtype=torch.bool, device="cuda") if results else None
        total += keys.numel()
        occ = (f.insertManySorted if sorted_ else f.insertMany)(keys, d_output=ok)
        assert occ == total == f.countOccupiedSlots()
        assert ok is None or bool(ok.all())
    st = f.stats()
    assert st["failed"] == st["lost"] == st["duplicates"] == 0
    assert st["primary"] + st["secondary"] + st["evicted_inserts"] == total
    for keys in batches:
        assert bool(f.containsMany(keys).all())
    for keys in batches:
        gone = torch.zeros(keys.numel(), dtype=torch.bool, device="cuda")
        total -= keys.numel()
        assert f.deleteMany(keys, gone) == total and bool(gone.all())
    assert int(f.table_image().to(torch.int32).sum()) == 0


@pytest.mark.parametrize("results", [False, True])
@pytest.mark.parametrize("kb,bits,bs,alt,slots,loads", [
    (8, 16, 16, "xor", 16, (0.5,)),                    # one bucket
    (8, 16, 16, "xor", 1 << 8, (0.5, 0.3)),            # one segment
    (8, 16, 16, "xor", 1 << 14, (0.0625, 0.7)),        # exactly one key per bucket
    (4, 16, 16, "xor", 1 << 20, (0.5, 0.4)),           # one pass, a table that is not empty
    (8, 8, 16, "xor", 1 << 20, (0.9,)),
    (8, 8, 8, "xor", 1 << 18, (0.5, 0.3)),             # 8-byte buckets
    (8, 16, 4, "xor", 1 << 18, (0.85,)),
    (8, 32, 8, "xor", 1 << 19, (0.4, 0.45)),           # 8-byte entries
    (4, 32, 2, "xor", 1 << 16, (0.55,)),
    (8, 16, 16, "addsub", 1_000_003, (0.6, 0.3)),      # partial last segment, primary buckets in one half
    (4, 16, 16, "offset", 777_777, (0.5, 0.4)),
    (8, 16, 16, "offset", 100, (0.7,)),
    (8, 16, 16, "xor", 1 << 25, (0.1, 0.2)),           # two passes, 4-byte entries between them
    (8, 32, 8, "xor", 1 << 24, (0.3,)),                # two passes, 8-byte entries
    (8, 16, 16, "offset", 20_000_000, (0.2,)),         # two passes, partial last segment
])
def test_binned_insert_stores_exactly_the_batch(cfb, orc, kb, bits, bs, alt, slots, loads, results):
    policy = cfb.EvictionPolicy(int(results))
    cfg = cfb.CuckooConfig(T="uint64" if kb == 8 else "uint32", bitsPerTag=bits, bucketSize=bs, maxEvictions=500,
                           AltBucketPolicy=POLICY[alt], evictionPolicy=policy)
    f = cfb.CuckooFilter(cfg, slots)
    cap, batches, at = f.capacity(), [], 0
    for load in loads:
        n = max(f.getNumBuckets(), int(load * cap))
        keys = orc.splitmix64(11 + bits + bs, n, first=at)
        at += n
        if kb == 4:
            keys = keys.astype(np.uint32)
        batches.append(dev(keys))
    filled_and_emptied(cfb, f, batches, results, sorted_=bits == 32)
    f.close()


def test_binned_insert_with_entries_of_both_widths(cfb, orc):
    """A 1 GiB table: 8-byte entries between the passes, 4-byte ones in the segments' bins."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 29)
    n = f.getNumBuckets()
    filled_and_emptied(cfb, f, [dev(orc.splitmix64(5, n + 1)), dev(orc.splitmix64(5, n + 777, first=n + 1))], False)
    f.close()


@pytest.mark.parametrize("kb,bits,bs,slots,hot,copies,limit", [
    (8, 16, 16, 1 << 16, 1, 5000, 0),       # one value repeated past its segment's bin
    (8, 16, 16, 1 << 16, 40, 300, 0),
    (8, 16, 16, 1 << 25, 3, 700_000, 0),    # past a first-pass bin and past a segment's bin
    (8, 32, 8, 1 << 24, 1, 1_800_000, 0),
    (8, 32, 8, 1 << 24, 1, 1_800_000, 80),  # a list of half the batch, too short: the segment-staged path
    (8, 32, 8, 1 << 24, 1, 300_000, 80),    # a list of half the batch that suffices
])
@pytest.mark.parametrize("results", [False, True])
def test_binned_insert_of_repeated_keys(cfb, orc, kb, bits, bs, slots, hot, copies, limit, results):
    """Batches that do not hash evenly: what fits is stored, every other key of the
    batch is, and the counters and flags agree with the table."""
    if limit and results:
        limit = 120
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=bits, bucketSize=bs, maxEvictions=4,
                           evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, slots)
    if limit:
        f.setOption(cfb.OPT_WORKSPACE_LIMIT, limit << 20)
    rest = orc.splitmix64(21, max(f.getNumBuckets(), int(0.15 * slots)))
    hots = orc.splitmix64(22, hot)
    keys = np.concatenate([np.repeat(hots, copies), rest])
    keys = keys[np.random.default_rng(4).permutation(len(keys))]
    d = dev(keys)
    ok = torch.zeros(len(keys), dtype=torch.bool, device="cuda") if results else None
    occ = f.insertMany(d, d_output=ok)
    st = f.stats()
    assert occ == f.countOccupiedSlots() == len(keys) - st["failed"] - st["lost"] + st["duplicates"]
    assert st["failed"] >= hot * (copies - 2 * bs) - st["lost"]
    assert bool(f.containsMany(dev(hots)).all())
    if results:
        assert int(ok.sum()) == len(keys) - st["failed"]
    if st["lost"] == 0:
        # a key fails only when both its buckets are buckets of repeated values, which
        # are full of them: any other key's second bucket has room at this load
        c = cfb.CuckooFilter.getCandidateBuckets(cfg, rest, f.getNumBuckets())
        h = cfb.CuckooFilter.getCandidateBuckets(cfg, hots, f.getNumBuckets())
        full = np.unique(np.concatenate(h[:2]))
        hopeless = np.isin(c[0], full) & np.isin(c[1], full)
        assert np.all(host_u8(f.containsMany(dev(rest))).astype(bool) | hopeless)
    f.close()


@pytest.mark.parametrize("results", [False, True])
@pytest.mark.parametrize("bits,slots,n,copies,dfs", [
    (16, 1 << 16, 9000, 5000, True),             # walks over a short list
    (16, 1 << 24, 3 << 20, 1 << 20, True),
    (8, 1 << 20, 1 << 19, 1 << 18, False),       # eviction lanes
    (8, 1 << 27, (1 << 25) + 4096, 5000, False), # the lockstep pass
])
def test_binned_insert_evicts_beside_stored_entries(cfb, orc, bits, slots, n, copies, dfs, results):
    """The eviction kernels on a list where entries without room in a bin have been
    stored (and zeroed) between ones that have not."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=bits, bucketSize=16, maxEvictions=4,
                           evictionPolicy=cfb.EvictionPolicy.DFS if dfs else cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, slots)
    rest = dev(orc.splitmix64(41, n))
    hot = dev(orc.splitmix64(42, 1))
    near = f.getNumBuckets() // 256  # keys of the repeated key's segment at least get no room in its bin
    keys = torch.cat([hot.expand(copies), rest])
    keys = keys[torch.randperm(keys.numel(), device="cuda", generator=torch.Generator("cuda").manual_seed(near))].contiguous()
    ok = torch.zeros(keys.numel(), dtype=torch.bool, device="cuda") if results else None
    occ = f.insertMany(keys, d_output=ok)
    st = f.stats()
    assert occ == f.countOccupiedSlots() == keys.numel() - st["failed"] - st["lost"] + st["duplicates"]
    assert st["primary"] + st["secondary"] + st["evicted_inserts"] == keys.numel()
    assert copies - 32 - st["lost"] <= st["failed"] <= copies
    assert ok is None or int(ok.sum()) == keys.numel() - st["failed"]
    assert bool(f.containsMany(hot).all())
    if st["lost"] == 0:
        assert bool(f.containsMany(rest).all())
    f.close()


def launches_of(cfb, f, call):
    before = cfb.launch_count()
    call()
    return cfb.launch_count() - before


def test_options_of_the_segment_path_are_obeyed(cfb, orc):
    """CF_STAGING_SEGMENT and CF_OPT_ROUND2_SEGMENTED_MIN_KEYS select and steer the
    segment-staged insert at one key per bucket and more, where automatic inserts are binned."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 21)
    d = dev(orc.splitmix64(341, int(0.8 * f.capacity())))
    n = {}
    for name, opts in {"auto": {}, "segment": {cfb.OPT_STAGING: cfb.STAGING_SEGMENT},
                       "round2 staged": {cfb.OPT_ROUND2_SEGMENTED_MIN_KEYS: 1},
                       "round2 random": {cfb.OPT_ROUND2_SEGMENTED_MIN_KEYS: cfb.NEVER}}.items():
        f.clear()
        for o, v in opts.items():
            f.setOption(o, v)
        n[name] = launches_of(cfb, f, lambda: f.insertMany(d))
        assert f.countOccupiedSlots() == d.numel() and bool(f.containsMany(d).all())
        f.setOption(cfb.OPT_STAGING, cfb.STAGING_AUTO)
        f.setOption(cfb.OPT_ROUND2_SEGMENTED_MIN_KEYS, 0)
    # one random pass in the place of two more sorted rounds and three eviction kernels
    assert n["round2 random"] < n["round2 staged"] == n["segment"] != n["auto"], n
    f.close()


@pytest.mark.parametrize("dfs", [False, True])
@pytest.mark.parametrize("results", [False, True])
@pytest.mark.parametrize("kb,bits,bs,loads,limit", [
    (8, 8, 16, (0.5, 0.4), 0), (8, 16, 16, (0.9,), 0), (4, 16, 16, (0.5, 0.4), 0), (8, 16, 4, (0.5, 0.35), 0),
    (8, 8, 8, (0.9,), 0),
    (8, 16, 16, (0.6, 0.3), 9), (4, 8, 16, (0.9,), 9),  # too little workspace to bin, chunks past a key per bucket
])
def test_segment_staged_inserts_where_binned_ones_would_do(cfb, orc, kb, bits, bs, loads, limit, results, dfs):
    """The path that binned inserts fall back on: narrow entries, ranked claims in three
    rounds, on an empty table and a filled one, with and without results."""
    cfg = cfb.CuckooConfig(T="uint64" if kb == 8 else "uint32", bitsPerTag=bits, bucketSize=bs, maxEvictions=500,
                           evictionPolicy=cfb.EvictionPolicy.DFS if dfs else cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 20)
    if limit:
        f.setOption(cfb.OPT_WORKSPACE_LIMIT, limit << 20)
    else:
        f.setOption(cfb.OPT_STAGING, cfb.STAGING_SEGMENT)
    at, batches = 0, []
    for load in loads:
        n = int(load * f.capacity())
        keys = orc.splitmix64(350 + bits + bs, n, first=at)
        at += n
        batches.append(dev(keys.astype(np.uint32) if kb == 4 else keys))
    filled_and_emptied(cfb, f, batches, results, sorted_=True)
    assert f.getOption(cfb.OPT_WORKSPACE_BYTES) <= (limit << 20 or 1 << 30)
    f.close()


@pytest.mark.parametrize("results,limit", [(False, 49 << 20), (True, 66 << 20)])
@pytest.mark.parametrize("dfs", [False, True])
def test_binned_insert_past_a_half_length_list(cfb, orc, results, limit, dfs):
    """A list of half the batch that is long enough for the first round and not for
    the second: every key's primary bucket is full, and every alternate bucket
    lies in a quarter of the table that is empty and has room for all of them."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=32, bucketSize=8, maxEvictions=100,
                           evictionPolicy=cfb.EvictionPolicy.DFS if dfs else cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 24)
    nb = f.getNumBuckets()
    image = np.zeros((nb, 8), np.uint32)
    image[nb // 4:] = np.arange(1, 6 * nb + 1, dtype=np.uint32).reshape(-1, 8) | np.uint32(1)
    f.load_table(torch.from_numpy(image.view(np.uint8).reshape(-1)).cuda())
    full = f.occupiedSlots()
    assert full == 6 * nb
    pool = orc.splitmix64(51, 12 << 20)
    i1, i2, _ = cfb.CuckooFilter.getCandidateBuckets(cfg, pool, nb)
    keys = pool[(i1 >= nb // 4) & (i2 < nb // 4)]
    assert len(keys) >= nb
    d = dev(keys[:nb])
    f.setOption(cfb.OPT_WORKSPACE_LIMIT, limit)
    ok = torch.zeros(nb, dtype=torch.bool, device="cuda") if results else None
    occ = f.insertMany(d, d_output=ok)
    st = f.stats()
    assert occ == full + nb == f.countOccupiedSlots() and st["failed"] == st["lost"] == st["duplicates"] == 0, st
    assert st["primary"] + st["secondary"] + st["evicted_inserts"] == nb
    assert ok is None or bool(ok.all())
    assert bool(f.containsMany(d).all())
    f.close()


@pytest.mark.parametrize("alt,load,cap", [("xor", 0.6, 0), ("addsub", 0.95, 0), ("xor", 0.6, 2)])
def test_large_binned_inserts_keep_their_rounds(cfb, alt, load, cap):
    """Fills of 2^27 keys and more, where a list of half the batch would do and where the
    first round leaves more than that: three rounds of binning all the same."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, AltBucketPolicy=POLICY[alt],
                           evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, int((1 << 27) / load) + (1 << 20) if alt != "xor" else 1 << 28)
    if cap:
        f.setOption(cfb.OPT_ROUND1_CAP, cap)
    n = (1 << 27) + 12345
    keys = torch.randint(-2 ** 63, 2 ** 63 - 1, (n,), device="cuda", generator=torch.Generator("cuda").manual_seed(9))
    launches = launches_of(cfb, f, lambda: f.insertMany(keys))
    assert launches >= 13, launches  # 3 x (2 binning passes, insert), then the lists
    st = f.stats()
    assert f.occupiedSlots() == f.countOccupiedSlots() == n and st["failed"] == st["lost"] == st["duplicates"] == 0
    assert bool(f.containsMany(keys).all())
    f.close()


@pytest.mark.parametrize("bits,bs", [(8, 16), (16, 16), (32, 8)])
@pytest.mark.parametrize("kpt", [1, 2, 4, 8])
def test_set_items_that_end_inside_a_thread(cfb, orc, bits, bs, kpt):
    """Items of 0 to 40 keys, so that a thread's keys, a warp's and a tile's belong
    to several filters, with one item of a filter outside the set; every filter
    ends up as its own keys inserted into the oracle would leave it."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=bits, bucketSize=bs, evictionPolicy=cfb.EvictionPolicy.BFS)
    nf = 48
    fs = cfb.CuckooFilterSet(cfg, [512] * nf)
    rng = np.random.default_rng(kpt)
    sizes = rng.choice([0, 1, 2, 3, 5, 8, 31, 33, 40], 400)
    filt = rng.integers(0, nf, 400).astype(np.int32)
    filt[200] = nf + 7
    sizes[200] = 3
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(offs[-1])
    keys = orc.splitmix64(31, n)
    for op in (cfb.SET_INSERT, cfb.SET_CONTAINS, cfb.SET_DELETE):
        fs.set_launch(op, 128, kpt)
    owner = np.repeat(filt, sizes)
    ok = owner < nf
    d, o, w = dev(keys), torch.from_numpy(offs).cuda(), torch.from_numpy(filt).cuda()
    res = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    fs.insert_async(d, o, w, res)
    with pytest.raises(cfb.CuckooError):
        fs.sync()
    got = res.cpu().numpy()
    assert np.array_equal(got, ok.astype(np.uint8))  # at most 300 keys in 512 slots: none fails
    occ = fs.occupied()
    for i in range(nf):
        assert occ[i] == int((owner == i).sum()) == fs.stats(i)["occupied"]
        assert fs.stats(i)["primary"] + fs.stats(i)["secondary"] + fs.stats(i)["evicted_inserts"] == occ[i]
    fs.contains_async(d, o, w, res)
    assert np.array_equal(res.cpu().numpy(), ok.astype(np.uint8))
    half = np.arange(n) % 2 == 0  # delete the even keys, as items of the same filters
    o2 = torch.from_numpy(np.concatenate([[0], np.cumsum(half)])[offs].astype(np.int64)).cuda()
    gone = torch.full((int(half.sum()),), 7, dtype=torch.uint8, device="cuda")
    fs.delete_async(dev(keys[half]), o2, w, gone)
    assert np.array_equal(gone.cpu().numpy(), ok[half].astype(np.uint8))
    occ = fs.occupied()
    for i in range(nf):
        assert occ[i] == int((owner[~half] == i).sum())
    fs.contains_async(dev(keys[~half]), torch.from_numpy(np.concatenate([[0], np.cumsum(~half)])[offs].astype(np.int64)).cuda(),
                      w, res[:int((~half).sum())])
    assert np.array_equal(res[:int((~half).sum())].cpu().numpy(), ok[~half].astype(np.uint8))


@pytest.mark.parametrize("n_items", [1, 2, 31, 33, 1025, 40_000])
@pytest.mark.parametrize("block,kpt", [(32, 1), (128, 8), (512, 4)])
def test_set_of_many_small_items(cfb, orc, n_items, block, kpt):
    """Items of 0 to 5 keys, many of them empty, a filter in several items: counters,
    results and occupancy of every filter."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    nf = max(1, n_items // 2)
    fs = cfb.CuckooFilterSet(cfg, [64] * nf)
    rng = np.random.default_rng(n_items + kpt)
    sizes = rng.choice([0, 0, 1, 2, 3, 5], n_items)
    sizes[-1] = 4
    filt = rng.permutation(n_items).astype(np.int32) % nf  # at most 3 items, 15 keys, per filter
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    keys, owner = orc.splitmix64(401, int(offs[-1])), np.repeat(filt, sizes)
    for op in (cfb.SET_INSERT, cfb.SET_CONTAINS, cfb.SET_DELETE):
        fs.set_launch(op, block, kpt)
    d, o, w = dev(keys), torch.from_numpy(offs).cuda(), torch.from_numpy(filt).cuda()
    res = torch.full((len(keys),), 7, dtype=torch.uint8, device="cuda")
    want = np.bincount(owner, minlength=nf)
    fs.insert_async(d, o, w, res)
    fs.sync()
    assert bool((res == 1).all()) and np.array_equal(fs.occupied(), want)
    for i in rng.integers(0, nf, 50):
        st = fs.stats(int(i))
        assert st["primary"] + st["secondary"] == want[i] and st["evicted_inserts"] == 0
    fs.contains_async(d, o, w, res.fill_(7))
    fs.sync()
    assert bool((res == 1).all())
    fs.delete_async(d, o, w, res.fill_(7))
    fs.sync()
    assert bool((res == 1).all()) and int(fs.occupied().sum()) == 0
    for i in rng.integers(0, nf, 50):
        assert fs.stats(int(i))["removed"] == want[i]
    fs.delete_async(d, o, w, res)
    fs.sync()
    assert int(res.sum()) == 0 and int(fs.occupied().sum()) == 0


@pytest.mark.parametrize("kb,bits,bs,load", [(8, 16, 16, 0.99), (4, 8, 16, 0.98), (8, 8, 8, 0.95), (8, 32, 8, 0.97),
                                             (8, 16, 4, 0.93), (8, 32, 2, 0.86)])
def test_short_eviction_lists(cfb, orc, kb, bits, bs, load):
    """A fill past the load where keys begin to fail, with as many eviction lanes
    per key as the geometry has candidates: flags, counters, chain histogram and
    table agree, and every stored key can be taken out again."""
    cfg = cfb.CuckooConfig(T="uint64" if kb == 8 else "uint32", bitsPerTag=bits, bucketSize=bs, maxEvictions=200,
                           evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 18)
    f.setOption(cfb.OPT_CHAIN_HISTOGRAM, 1)
    keys = orc.splitmix64(61 + bits + bs, int(load * f.capacity()))
    if kb == 4:
        keys = keys.astype(np.uint32)
    d = dev(keys)
    ok = torch.zeros(len(keys), dtype=torch.bool, device="cuda")
    occ = f.insertMany(d, d_output=ok)
    st = f.stats()
    stored = int(ok.sum())
    assert stored == len(keys) - st["failed"]
    assert occ == f.countOccupiedSlots() == stored - st["lost"] + st["duplicates"]
    assert st["evicted_inserts"] > 0 and st["evictions"] > 0
    assert int(f.chainHistogram().sum()) == st["evicted_inserts"] - st["failed"]
    if st["lost"] == st["duplicates"] == 0:
        assert bool(f.containsMany(d[ok]).all())
        gone = torch.zeros(stored, dtype=torch.bool, device="cuda")
        assert f.deleteMany(d[ok], gone) == 0 and bool(gone.all())
        assert int(f.table_image().to(torch.int32).sum()) == 0
    f.close()


@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 20) - 1, 1 << 20])
@pytest.mark.parametrize("load", [0.5, 0.8])
def test_insertMany_route_by_batch_size(cfb, orc, n, load):
    """Around the batch sizes where insertMany changes from random probes to
    binning, for batches that fill the table beyond three quarters and not."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, AltBucketPolicy=POLICY["offset"],
                           evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, int(n / load))
    keys = orc.splitmix64(71, n)
    before = cfb.launch_count()
    f.insertMany(dev(keys))
    launches = cfb.launch_count() - before
    staged = n >= (1 << 17 if load > 0.75 else 1 << 20)
    assert (launches >= 8) == staged and (launches <= 2) == (not staged), launches
    f.clear()
    filled_and_emptied(cfb, f, [dev(keys)], False)
    f.close()


@pytest.mark.parametrize("n", [1, 31, 512, 513, 40_000])
def test_counts_of_synchronous_calls_from_several_threads(cfb, orc, n):
    """The count a synchronous random insert or delete returns is written by its
    own last CTA: threads that work on one filter at the same time, on streams of
    their own, each get a count that lies between what was there before and after,
    and the last ones agree with the table."""
    import threading

    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 20)
    rounds, nt = 6, 4
    keys = [dev(orc.splitmix64(80 + i, n)) for i in range(nt)]
    streams = [torch.cuda.Stream() for _ in range(nt)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            with torch.cuda.stream(streams[i]):
                for _ in range(rounds):
                    a = f.insertMany(keys[i])
                    b = f.deleteMany(keys[i])
                    if not (n <= a <= nt * n and 0 <= b <= (nt - 1) * n):
                        bad.append((i, a, b))
        except Exception as e:  # noqa: BLE001
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(nt)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    assert f.occupiedSlots() == f.countOccupiedSlots() == 0
    assert f.insertMany(keys[0]) == n == f.occupiedSlots()
    assert f.insertMany(keys[0][:0]) == n and f.deleteMany(keys[0][:0]) == n  # nothing to launch
    assert f.deleteMany(keys[0]) == 0
    f.close()


def test_counts_while_a_long_call_is_in_flight(cfb, orc):
    """One thread makes hundreds of small synchronous calls on a high-priority
    stream while another's large deletes run (of keys that are not there): every
    count is the call's own, and none is stale afterwards."""
    import threading

    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=32, bucketSize=8, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 28)
    absent = dev(orc.splitmix64(101, 1 << 24)).repeat(8)
    small = dev(orc.splitmix64(102, 1000))
    torch.cuda.synchronize()
    bad, done, long_counts = [], threading.Event(), []

    def long_calls():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    long_counts.append(f.deleteMany(absent))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))
        done.set()

    t = threading.Thread(target=long_calls)
    t.start()
    stored = 0
    with torch.cuda.stream(torch.cuda.Stream(priority=-1)):
        while (not done.is_set() or stored < 300) and stored < 800:
            got = f.insertMany(small[stored:stored + 1])
            stored += 1
            if got != stored:
                bad.append((stored, got))
    t.join()
    for _ in range(130):
        got = f.insertMany(small[stored:stored + 1])
        stored += 1
        if got != stored:
            bad.append((stored, got))
    assert not bad, bad[:5]
    assert len(long_counts) == 8 and long_counts == sorted(long_counts) and 0 <= long_counts[0] <= long_counts[-1] <= stored
    assert f.occupiedSlots() == f.countOccupiedSlots() == stored
    f.close()


def test_counts_of_more_calls_than_rows(cfb, orc):
    """More threads than a filter has rows of published counters."""
    import threading

    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 20)
    n, rounds, nt = 513, 4, 80
    keys = [dev(orc.splitmix64(200 + i, n)) for i in range(nt)]
    streams = [torch.cuda.Stream() for _ in range(nt)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            for _ in range(rounds):
                a = f.insertMany(keys[i], stream=streams[i])
                b = f.deleteMany(keys[i], stream=streams[i])
                if not (n <= a <= nt * n and 0 <= b <= (nt - 1) * n):
                    bad.append((i, a, b))
        except Exception as e:  # noqa: BLE001
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(nt)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:5]
    for k in range(130):
        assert f.insertMany(keys[k % nt][k:k + 1]) == k + 1
    f.close()


@pytest.mark.parametrize("staging", ["auto", "segment", "region"])
@pytest.mark.parametrize("results", [False, True])
def test_staged_batches_on_two_streams(cfb, orc, staging, results):
    """Asynchronous staged batches of one filter on several streams, with nothing
    between them: they share one workspace and the table, and leave what they
    would leave one after the other.  So do calls that follow one on another stream."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 24)
    f.setOption(cfb.OPT_STAGING, {"auto": cfb.STAGING_AUTO, "segment": cfb.STAGING_SEGMENT, "region": cfb.STAGING_REGION}[staging])
    n = 5 << 20
    a, b, few = dev(orc.splitmix64(301, n)), dev(orc.splitmix64(302, n + 77)), dev(orc.splitmix64(303, 1000))
    oks = [torch.full((k.numel(),), 7, dtype=torch.uint8, device="cuda") if results else None for k in (a, b, few)]
    s1, s2, s3 = (torch.cuda.Stream() for _ in range(3))
    for _ in range(3):
        f.clear()
        torch.cuda.synchronize()
        f.insertManyAsync(a, stream=s1, d_output=oks[0])
        f.insertManyAsync(b, stream=s2, d_output=oks[1])
        f.insertManyAsync(few, stream=s3, d_output=oks[2])  # (at random, left to itself)
        f.deleteManyAsync(few, stream=s3)
        torch.cuda.synchronize()
        assert f.occupiedSlots() == f.countOccupiedSlots() == a.numel() + b.numel()
        st = f.stats()
        assert st["failed"] == st["lost"] == st["duplicates"] == 0 and st["removed"] == 1000
        assert bool(f.containsMany(a).all()) and bool(f.containsMany(b).all())
        for k, ok in zip((a, b, few), oks):
            assert ok is None or int(ok.sum()) == k.numel()
        f.insertManyAsync(few, stream=s2)
        f.deleteManyAsync(b, stream=s3)
        f.deleteManyAsync(a, stream=s1)
        torch.cuda.synchronize()
        assert f.occupiedSlots() == f.countOccupiedSlots() == 1000
        f.insertManyAsync(a, stream=s1)
        f.clear(stream=s2)
        torch.cuda.synchronize()
        assert f.occupiedSlots() == f.countOccupiedSlots() == 0
    f.close()


def test_capture_beside_an_asynchronous_staged_batch(cfb, orc):
    """Random calls are captured and replayed on one stream although the last staged
    batch, on another, has only been waited for by the caller."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 22)
    many, few = dev(orc.splitmix64(361, 2 << 20)), dev(orc.splitmix64(362, 1000))
    found, gone = (torch.zeros(1000, dtype=torch.bool, device="cuda") for _ in range(2))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    f.insertMany(few), f.containsMany(few, found), f.deleteMany(few, gone)  # modules loaded
    torch.cuda.synchronize()
    f.insertManyAsync(many, stream=s1)
    torch.cuda.synchronize()
    found.zero_(), gone.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s2):
        f.insertManyAsync(few, stream=s2)
        f.containsManyAsync(few, found, stream=s2)
        f.deleteManyAsync(few, gone, stream=s2)
    assert f.occupiedSlots() == many.numel()  # nothing has run yet
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert bool(found.all()) and bool(gone.all())
        assert f.occupiedSlots() == f.countOccupiedSlots() == many.numel()
        found.zero_(), gone.zero_()
    assert bool(f.containsMany(many).all())
    f.close()


def test_counters_read_after_an_asynchronous_staged_batch(cfb, orc):
    """Every read of the counters waits for the staged batch before it, on a stream
    that the legacy default stream does not wait for by itself."""
    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 26)
    f.setOption(cfb.OPT_CHAIN_HISTOGRAM, 1)
    d = dev(orc.splitmix64(331, int(0.9 * f.capacity())))
    n = d.numel()
    s = torch.cuda.Stream()
    f.insertMany(d)  # the workspace exists
    reads = {"occupied": lambda: f.occupiedSlots() == n,
             "slots": lambda: f.countOccupiedSlots() == n,
             "stats": lambda: (lambda st: st["primary"] + st["secondary"] + st["evicted_inserts"] == n)(f.stats()),
             "chains": lambda: int(f.chainHistogram().sum()) == f.stats()["evicted_inserts"] > 0,
             "reset": lambda: f.resetEvictionCount() is None and f.evictionCount() == 0}
    for name, read in reads.items():
        f.clear()
        torch.cuda.synchronize()
        f.insertManyAsync(d, stream=s)
        assert read(), name
        torch.cuda.synchronize()
        assert f.occupiedSlots() == n and (name != "reset" or f.evictionCount() == 0)
    f.close()


def test_staged_batches_of_several_threads(cfb, orc):
    """Threads that insert and delete staged batches of one filter at the same time, the
    workspace growing between them; every count lies between what other threads can leave."""
    import threading

    cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
    f = cfb.CuckooFilter(cfg, 1 << 23)
    sizes = [1 << 20, (1 << 20) + 5, 3 << 19, 7 << 18]
    keys = [dev(orc.splitmix64(310 + i, n)) for i, n in enumerate(sizes)]
    streams = [torch.cuda.Stream() for _ in sizes]
    f.setOption(cfb.OPT_SEGMENTED_MIN_KEYS, 1)  # deletes too
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            for r in range(4):
                a = f.insertMany(keys[i], stream=streams[i])
                if r & 1:
                    f.deleteManyAsync(keys[i], stream=streams[i])
                    b = 0
                else:
                    b = f.deleteMany(keys[i], stream=streams[i])
                if not (sizes[i] <= a <= sum(sizes) and 0 <= b <= sum(sizes) - sizes[i]):
                    bad.append((i, a, b))
        except Exception as e:  # noqa: BLE001
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not bad, bad[:5]
    st = f.stats()
    assert st["failed"] == st["lost"] == st["duplicates"] == 0
    assert f.occupiedSlots() == f.countOccupiedSlots() == 0
    assert f.insertMany(keys[0]) == sizes[0] and bool(f.containsMany(keys[0]).all())
    f.close()


FLUSH = r"""
#include <cstdio>
#include "cf_kernels.cuh"
__global__ void add(unsigned long long* ctr, int32_t big) {
    const int32_t t = static_cast<int32_t>(threadIdx.x);
    cfb::flush_counters(ctr, {{2, big - t}, {0, -big}, {1, (t & 1) ? 5 : -7}, {3, 0}});
}
int main() {
    unsigned long long* c;
    if (cudaMallocManaged(&c, 4 * sizeof *c) != cudaSuccess) return 2;
    for (int threads : {32, 96, 256, 512, 1024})
        for (int32_t big : {3, 1 << 30, 0x7fffffff}) {
            for (int i = 0; i < 4; ++i) c[i] = 1000;
            add<<<3, threads>>>(c, big);
            if (cudaDeviceSynchronize() != cudaSuccess) return 3;
            const long long n = 3ll * threads, tri = 3ll * threads * (threads - 1) / 2;
            const long long want[4] = {1000 - n * big, 1000 - n, 1000 + n * big - tri, 1000};
            for (int i = 0; i < 4; ++i)
                if (static_cast<long long>(c[i]) != want[i])
                    return printf("%d threads, counter %d: %lld, not %lld\n", threads, i, (long long)c[i], want[i]), 1;
        }
    return 0;
}
"""


def test_counter_sums_past_32_bits(cfb, tmp_path):
    """A CTA's sums of its threads' counts are exact however large and of whatever sign."""
    import subprocess

    pkg = os.path.dirname(cfb.__file__)
    sys.path.insert(0, pkg)
    import build

    src, exe = tmp_path / "flush.cu", tmp_path / "flush"
    src.write_text(FLUSH)
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I" + os.path.join(pkg, "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


CAPTURE = """
import __graft_entry__, oracle, torch
cfb = __graft_entry__.package()
cfg = cfb.CuckooConfig(T="uint64", bitsPerTag=16, bucketSize=16, evictionPolicy=cfb.EvictionPolicy.BFS)
f = cfb.CuckooFilter(cfg, 1 << 18)
keys = torch.from_numpy(oracle.splitmix64(91, int(0.9 * f.capacity())).view("int64")).cuda()
n = keys.numel()
f.insertMany(keys)  # the workspace exists
f.clear()
s = torch.cuda.Stream()
s.wait_stream(torch.cuda.current_stream())
refused = False
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=s):
        f.insertManyAsync(keys, stream=s)
except Exception:
    refused = True
torch.cuda.synchronize()
try:
    f.containsMany(keys)  # the CUDA runtime hands the refusal to the next call that asks for errors
except cfb.CuckooError:
    pass
f.clear()
assert refused and f.insertMany(keys) == n == f.countOccupiedSlots() and bool(f.containsMany(keys).all())
print("refused, and the filter works on")
"""


def test_binned_insert_is_refused_under_capture(cfb, orc):
    """A captured fill would replay with what was known of the table at capture
    time, so it ends in an error, and the filter works on afterwards.  (In a
    process of its own: a capture that fails leaves torch's allocator changed.)"""
    import subprocess

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "works on" in r.stdout, r.stdout + r.stderr
