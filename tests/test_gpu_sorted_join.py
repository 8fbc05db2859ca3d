"""The sort-merge names' counting sort at the edges of a chunk's layout:
chunks around 2^13 slots, one or two chunks a partition, runs of equal keys
longer than a chunk, keys that agree in their low or high bits, every fan-out,
materialisation.  Whole numbers: exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def keys(kind, n, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(n, dtype=np.uint64)
    if kind == "spread":
        k = rng.integers(0, 1 << 32, size=n, dtype=np.uint64)
    elif kind == "low_equal":
        k = (k << np.uint64(14)) & np.uint64(0xFFFFFFFF)
    elif kind == "high_equal":
        k = k % np.uint64(1 << 13) + np.uint64(0xFFFFE000)
    elif kind == "one_key":
        k = np.full(n, 0xFFFFFFFF, np.uint64)
    return rng.permutation(k).astype(np.uint32)


@pytest.mark.parametrize("kind", ["dense", "spread", "low_equal", "high_equal", "one_key"])
@pytest.mark.parametrize("n", [1, 2, 511, 8191, 8193, 16384, 17281, 17409, 40000])
def test_chunk_edges(oracle, kind, n):
    k = keys(kind, n, n)
    S = adb.tuples(np.concatenate([k[:3000], keys("spread", 100, 1)]))
    R = adb.tuples(k)
    got = adb.join("m-way", R, S, adb.default_params(part_fanout=2))
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("fanout", [2, 3, 64, 512, 513, 1024, 4096, 1 << 15, 1 << 16, 1 << 20])
def test_every_fan_out(oracle, fanout):
    k = keys("spread", 60000, 5)
    k[::4] = k[1::4]
    R, S = adb.tuples(k), adb.tuples(np.random.default_rng(6).choice(k, 70001))
    got = adb.join("m-pass", R, S, adb.default_params(part_fanout=fanout))
    assert (got.count, got.checksum) == oracle.truth(R, S)


def test_materialise(oracle):
    R, S = adb.tuples(keys("high_equal", 20000, 7)), adb.tuples(keys("high_equal", 9001, 8))
    want = oracle.truth(R, S)
    dR, dS, dO = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S), adb.DeviceBuffer(8 * want[0])
    got = adb.join_materialize_device("m-way+skew", dR.ptr, len(R), dS.ptr, len(S), dO.ptr, want[0])
    assert (got.count, got.checksum) == want and got.materialized == want[0]
    rows = dO.to_host(np.uint64, want[0])
    per_key = np.bincount(R["key"] - np.uint32(0xFFFFE000), minlength=1 << 13)
    expect = np.repeat(S.view(np.uint64), per_key[S["key"] - np.uint32(0xFFFFE000)])
    assert np.array_equal(np.sort(rows), np.sort(expect))
    for b in (dR, dS, dO):
        b.close()
