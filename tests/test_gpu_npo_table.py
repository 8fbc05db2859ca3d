"""NPO's bucket table and its hand-over to the partitioned join: odd bucket
counts, full buckets that spill to the next (and around the table's end),
tuples equal to the empty marker, a large S, and the sizes either side of the
dispatch rule.  radix_bits = -1 forces the table.  Whole numbers: exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def fk(n_r, n_s, seed, dup=1):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << 32, size=max(1, n_r // dup), dtype=np.uint64).astype(np.uint32)
    k = rng.permutation(np.resize(k, n_r))
    R = adb.tuples(k, rng.integers(0, 1 << 32, size=n_r, dtype=np.uint64).astype(np.uint32))
    return R, adb.tuples(np.concatenate([rng.choice(k, n_s - n_s // 8), rng.integers(0, 1 << 32, size=n_s // 8,
                                                                                     dtype=np.uint64).astype(np.uint32)]))


@pytest.mark.parametrize("n_r", [1, 2, 3, 4, 5, 7, 8, 4093, 8193, 100003, (1 << 20) + 1])
@pytest.mark.parametrize("dup", [1, 5])
def test_table_sizes(oracle, n_r, dup):
    R, S = fk(n_r, 20011, n_r, dup)
    got = adb.join("NPO", R, S, adb.default_params(radix_bits=-1))
    assert (got.count, got.checksum) == oracle.truth(R, S)


def test_spilling_buckets_and_empty_marker(oracle):
    # keys whose hash is at the table's end: their buckets overflow and wrap to the first
    hk = np.arange(0xFFFFFFFF - 299, 0xFFFFFFFF, dtype=np.uint64)
    inv = pow(0x9E3779B1, -1, 1 << 32)
    top = ((hk * inv) & 0xFFFFFFFF).astype(np.uint32)
    R = adb.tuples(np.concatenate([np.repeat(top, 3), np.full(50, 0xFFFFFFFF, np.uint32)]))
    R["payload"][-20:] = 0xFFFFFFFF          # 20 tuples equal to the empty marker
    S = adb.tuples(np.concatenate([top, np.full(7, 0xFFFFFFFF, np.uint32), np.arange(100, dtype=np.uint32)]))
    got = adb.join("NPO", R, S, adb.default_params(radix_bits=-1))
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("n_r,n_s", [(7 << 19, 1 << 20), ((7 << 19) + 1, 1 << 20), (1 << 22, 1 << 23),
                                     (1 << 22, (1 << 23) - 1), ((1 << 22) + 3, 1 << 23), (1 << 24, 1 << 18)])
def test_hand_over_to_the_partitioned_join(oracle, n_r, n_s):
    R = adb.gen_pk(n_r, 5)
    R["key"] *= np.uint32(0x01000193)        # distinct keys over all 32 bits
    S = adb.gen_fk(n_s, R, 0.5, 6)
    got = adb.join("NPO", R, S)
    assert (got.count, got.checksum) == oracle.truth(R, S)


def test_low_bits_equal_stay_spread(oracle):
    # 2^16 keys x 64 tuples that agree in their low 16 bits: the hashed digits still split them
    n = 1 << 22
    k = (np.arange(n, dtype=np.uint32) & np.uint32(0xFFFF)) << np.uint32(16)
    R = adb.tuples(k)
    S = adb.tuples(k[:5000])
    got = adb.join("NPO", R, S)
    assert got.count == 5000 * 64
    assert (got.count, got.checksum) == oracle.truth(R, S)
