"""A rank of a sharded join holds the keys of one destination (adb_shard_split);
the tables and digits of its local join take the top bits of key * kHashMul.  The
two must not fix one another: the keys of one shard must spread over all of the
local join's partitions and buckets.

On the CPU a model of the joins' rules with the constant read from the source; on
the GPU the joins of one shard, right and not slower than those of all keys."""
import re
from pathlib import Path

import numpy as np
import pytest

import alliancedb_b200 as adb
from alliancedb_b200.dist import shard_of

SRC = (Path(adb.__file__).parent / "csrc" / "adb_common.cuh").read_text()
HASH = int(re.search(r"kHashMul = (0x[0-9A-Fa-f]+)u", SRC)[1], 16)


def test_the_split_rule():
    """Values of the rule worked out with Python's integers."""
    m = (1 << 32) - 1
    for key in (0, 1, 2, 0x7FFFFFFF, 0x9E3779B1, 0xFFFFFFFF):
        h = ((key ^ (key >> 16)) * 0x85EBCA6B) & m
        h = ((h ^ (h >> 13)) * 0xC2B2AE35) & m
        for dtype in (np.uint32, np.uint64, np.int64):
            for parts in (1, 3, 8, 32):
                assert shard_of(np.array([key], dtype), parts)[0] == h * parts >> 32


def one_shard(n, parts, sparse, seed=1):
    """About n keys, distinct, of destination parts / 2."""
    if sparse:
        k = np.random.default_rng(seed).integers(0, 1 << 32, n * parts + n // 8 * parts, dtype=np.uint64)
    else:
        k = np.arange(1, n * parts + 1, dtype=np.uint64)
    return np.unique(k[shard_of(k, parts) == parts // 2])


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("parts", [1, 2, 4, 8, 32])
def test_one_shards_keys_spread(parts, sparse):
    k = one_shard(20_000, parts, sparse)
    n, h = k.size, k * np.uint64(HASH) & np.uint64(0xFFFFFFFF)
    fill = np.bincount((h >> np.uint64(24)).astype(np.int64), minlength=256)     # 2^8 partitions
    # binomial at most: mean + 6 standard deviations
    assert fill.max() <= n / 256 + 6 * np.sqrt(n / 256)
    # NPO: buckets of four slots, three slots a tuple; what a bucket cannot hold walks on, twice around
    nb = (3 * n + 3) // 4
    load = np.bincount((h * np.uint64(nb) >> np.uint64(32)).astype(np.int64), minlength=nb)
    x = np.cumsum(np.concatenate([load, load]) - 4)
    walked = (x - np.minimum.accumulate(np.minimum(x, 0)))[nb:].sum()
    assert walked / n < 0.1     # 0.012 for random keys


@pytest.mark.gpu
@pytest.mark.parametrize("parts", [4, 8])
@pytest.mark.parametrize("algo,n,bits", [("NPO", 1 << 20, -1), ("NPO", (7 << 19) + 1, 0), ("m-way", 1 << 21, 0),
                                         ("PRO", 1 << 13, 0), ("NPO", 1 << 15, 0)])
def test_joins_of_one_shard(oracle, algo, n, bits, parts):
    p = adb.default_params(radix_bits=bits)
    ms = []
    for k in (one_shard(n, parts, True)[:n], one_shard(n, 1, True)[:n]):
        rng = np.random.default_rng(2)
        k = rng.permutation(k).astype(np.uint32)
        assert k.size == n
        R, S = adb.tuples(k), adb.tuples(rng.choice(k, 100_003))
        got, want = [adb.join(algo, R, S, p) for _ in range(4)], oracle.truth(R, S)
        assert all((g.count, g.checksum) == want for g in got)
        ms.append(min(g.ms_device for g in got))
    assert ms[0] < 3 * ms[1] + 0.05     # with one hash for both: NPO's table by orders of magnitude


@pytest.mark.gpu
def test_spilling_buckets_at_the_tables_end(oracle):
    # keys whose hash is at the table's end: their buckets overflow and wrap to the first
    hk = np.arange(0xFFFFFFFF - 299, 0xFFFFFFFF, dtype=np.uint64)
    top = (hk * np.uint64(pow(HASH, -1, 1 << 32)) & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    R = adb.tuples(np.concatenate([np.repeat(top, 3), np.full(50, 0xFFFFFFFF, np.uint32)]))
    R["payload"][-20:] = 0xFFFFFFFF          # 20 tuples equal to the empty marker
    S = adb.tuples(np.concatenate([top, np.full(7, 0xFFFFFFFF, np.uint32), np.arange(100, dtype=np.uint32)]))
    for bits in (-1, 5):
        got = adb.join("NPO", R, S, adb.default_params(radix_bits=bits))
        assert (got.count, got.checksum) == oracle.truth(R, S)
