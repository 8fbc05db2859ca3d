"""Materialisation through every kernel that has that form, seen by the launches
of the call: the small join, the partitioned joins with one and two passes
(chained, hashed and sorted), NPO's table and its regions.  All matches, fewer
rows than matches, none; rows as a multiset against the oracle's."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu

SMALL, TABLE = (1,), (2,)
ONE_PASS, TWO_PASSES = (4,), (7, 8)
ROUTES = [
    ("PRO", 9000, 30011, {}, SMALL),
    ("NPO", 9000, 30011, {}, SMALL),
    ("PRO", 9000, 30011, {"radix_bits": 1}, ONE_PASS),
    ("PRH", 90001, 50021, {"radix_bits": 9}, ONE_PASS),
    ("RJ_st", 90001, 50021, {"radix_bits": 12}, TWO_PASSES),
    ("NPO", 90001, 50021, {"radix_bits": -1}, TABLE),
    ("NPO", 90001, 50021, {"radix_bits": 4}, (4,)),
    ("m-way", 9000, 30011, {}, ONE_PASS),
    ("m-pass", 90001, 50021, {"part_fanout": 1 << 11}, TWO_PASSES),
    ("NPO", (7 << 19) + 1, 50021, {}, ONE_PASS),
    ("NPO", (1 << 22) + 1, 50021, {}, TWO_PASSES),
]


def relations(n_r, n_s, seed):
    """Keys over 32 bits, one to three times in R; a third of S matches nothing, a few rows hold one hot key."""
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << 32, size=n_r // 2 + 1, dtype=np.uint64).astype(np.uint32)
    r = rng.permutation(np.concatenate([k, k])[:n_r])
    s = np.where(rng.random(n_s) < 0.67, rng.choice(k, n_s), rng.integers(0, 1 << 32, size=n_s, dtype=np.uint64)).astype(np.uint32)
    s[rng.integers(0, n_s, n_s // 50)] = r[0]
    return adb.tuples(r), adb.tuples(s)


@pytest.mark.parametrize("algo,n_r,n_s,params,kernels", ROUTES)
def test_rows(oracle, algo, n_r, n_s, params, kernels):
    R, S = relations(n_r, n_s, n_r)
    want = oracle.truth(R, S)
    # an S row comes once per match: its matches from R's sorted keys
    rk = np.sort(R["key"])
    times = np.searchsorted(rk, S["key"], "right") - np.searchsorted(rk, S["key"], "left")
    rows = np.sort(np.repeat(S.view(np.uint64), times))
    assert rows.size == want[0]
    dR, dS, dO = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S), adb.DeviceBuffer(8 * rows.size + 8)
    try:
        for cap in (rows.size, rows.size // 3, 0):
            mark = np.array([0x5A5A5A5A5A5A5A5A], np.uint64)
            adb._check(adb.lib().adb_memcpy_h2d(dO.ptr + 8 * cap, mark.ctypes.data, 8))
            got = adb.join_materialize_device(algo, dR.ptr, n_r, dS.ptr, n_s, dO.ptr, cap, adb.default_params(**params))
            assert got.kernels in kernels
            assert (got.count, got.checksum) == want and got.materialized == cap
            out = dO.to_host(np.uint64, cap + 1)
            assert out[cap] == mark[0]                     # nothing past the capacity
            if cap == rows.size:
                assert np.array_equal(np.sort(out[:cap]), rows)
            else:                                           # no row more often than it is one
                v, c = np.unique(out[:cap], return_counts=True)
                at, end = np.searchsorted(rows, v), np.searchsorted(rows, v, "right")
                assert np.all(c <= end - at)
    finally:
        for b in (dR, dS, dO):
            b.close()


def test_one_row_with_many_matches(oracle):
    """Rows of one lane by the thousand, the others of its warp with none."""
    R = adb.tuples(np.full(7001, 9, np.uint32))
    S = adb.tuples(np.concatenate([np.arange(100, 131, dtype=np.uint32), [9], np.arange(200, 260, dtype=np.uint32)]))
    dR, dS, dO = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S), adb.DeviceBuffer(8 * 7001)
    for algo, params in (("PRO", {}), ("PRO", {"radix_bits": 2}), ("m-way", {}), ("NPO", {"radix_bits": -1})):
        got = adb.join_materialize_device(algo, dR.ptr, 7001, dS.ptr, len(S), dO.ptr, 7001, adb.default_params(**params))
        assert got.count == got.materialized == 7001
        assert np.all(dO.to_host(np.uint64, 7001) == S.view(np.uint64)[31])
    for b in (dR, dS, dO):
        b.close()
