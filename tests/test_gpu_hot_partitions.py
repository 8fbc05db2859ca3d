"""Partitions with hot keys on both sides: their S pages go to several items, each
R chunk against each of them once.  Counts and checksums exact; and the pairs of a
few keys must keep more than a few CTAs busy."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo,params", [("PRO", {"radix_bits": 1}), ("PRO", {"radix_bits": 9}), ("PRH", {"radix_bits": 11}),
                                         ("m-way", {}), ("m-pass", {"part_fanout": 1 << 11})])
@pytest.mark.parametrize("hot_r,hot_s", [(1, 1025), (1, 30_011), (8703, 1023), (8705, 1025), (18_001, 3_001), (3_001, 62_000)])
def test_hot_key_on_both_sides(oracle, algo, params, hot_r, hot_s):
    rng = np.random.default_rng(hot_r + hot_s)
    k = rng.permutation(1 << 20)[:20_011].astype(np.uint32) * np.uint32(4093) + np.uint32(1)
    r = rng.permutation(np.concatenate([k[1:], np.full(hot_r, k[0])]))
    s = rng.permutation(np.concatenate([rng.choice(k[1:], 40_009), np.full(hot_s, k[0])]))
    R, S = adb.tuples(r, rng.integers(0, 1 << 32, r.size, dtype=np.uint64).astype(np.uint32)), adb.tuples(s)
    got = adb.join(algo, R, S, adb.default_params(**params))
    assert (got.count, got.checksum) == oracle.truth(R, S)
    dO = adb.DeviceBuffer(8)
    dR, dS = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)
    got = adb.join_materialize_device(algo, dR.ptr, len(R), dS.ptr, len(S), dO.ptr, 1, adb.default_params(**params))
    assert (got.count, got.materialized) == (hot_r * hot_s + 40_009, 1)
    for b in (dO, dR, dS):
        b.close()


def test_eight_keys_fill_the_chip():
    """2^17 tuples of 8 keys a side, 2.1 G pairs: the partitioned joins next to the small one."""
    rng = np.random.default_rng(5)
    R, S = (adb.tuples(rng.integers(0, 8, 1 << 17).astype(np.uint32)) for _ in range(2))
    want = int((np.bincount(R["key"]).astype(np.int64) * np.bincount(S["key"])).sum())
    ms = {}
    for name, algo, params in (("small", "PRO", {}), ("chained", "PRO", {"radix_bits": 8}), ("sorted", "m-way", {})):
        got = [adb.join(algo, R, S, adb.default_params(**params)) for _ in range(3)]
        assert all(g.count == want and g.checksum == got[0].checksum for g in got)
        ms[name] = min(g.ms_device for g in got)
    assert max(ms.values()) < 5 * ms["small"], ms    # sorted 15 times with one item per partition
