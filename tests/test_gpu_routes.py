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
