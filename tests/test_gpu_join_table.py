"""The partitioned join's chained table at the edges of its shared-memory
layout: R chunks around 2^13 slots (where the bucket heads stop growing), every
count of consumed radix bits (the link bits of a linked key), one long chain,
and batched windows around the sizes that may go unpartitioned.  Whole
numbers: count and checksum are exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def spread(n, seed):
    """n distinct keys anywhere in 32 bits (the extremes among them)."""
    rng = np.random.default_rng(seed)
    k = np.unique(rng.integers(0, 1 << 32, size=n + n // 8 + 64, dtype=np.uint64).astype(np.uint32))
    k = rng.permutation(k)[:n]
    k[: min(2, n)] = np.array([0, 0xFFFFFFFF], np.uint32)[: min(2, n)]
    return k


@pytest.mark.parametrize("n", [16380, 16384, 17270, 17280, 17290, 17408, 17500])
def test_chunk_edges_two_partitions(oracle, n):
    # radix_bits = 1: two partitions of about n / 2 tuples, one or two chunks each
    rng = np.random.default_rng(n)
    k = spread(n, n)
    R, S = adb.tuples(k), adb.tuples(rng.choice(k, 3 * n))
    got = adb.join("PRO", R, S, adb.default_params(radix_bits=1))
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("bits", range(1, 16))
def test_every_link_width(oracle, bits):
    rng = np.random.default_rng(bits)
    k = spread(40009, bits)
    k[::3] = rng.choice(k, k[::3].size)      # repeated build keys as well
    R, S = adb.tuples(k), adb.tuples(np.concatenate([rng.choice(k, 50021), spread(1000, 99)]))
    got = adb.join("PRO", R, S, adb.default_params(radix_bits=bits))
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("n", [8192, 8640, 8705, 20000])
def test_one_chain(oracle, n):
    R = adb.tuples(np.full(n, 0x80000001, np.uint32))
    S = adb.tuples(np.array([0x80000001, 1, 0x80000001, 0xFFFFFFFF], np.uint32))
    got = adb.join("PRO", R, S, adb.default_params(radix_bits=1))
    assert got.count == 2 * n
    assert (got.count, got.checksum) == oracle.truth(R, S)


def test_unpartitioned_batch_windows(oracle):
    sizes = [1, 2, 3, 63, 64, 65, 4095, 4096, 4097, 8191, 8192, 8193, 9000]
    rng = np.random.default_rng(5)
    Rs = [adb.tuples(spread(n, 100 + n)) for n in sizes]
    Ss = [adb.tuples(rng.choice(r["key"], 2 * len(r) + 5)) for r in Rs]
    r_off = np.concatenate([[0], np.cumsum([len(r) for r in Rs])]).astype(np.uint64)
    s_off = np.concatenate([[0], np.cumsum([len(s) for s in Ss])]).astype(np.uint64)
    dR, dS = adb.DeviceBuffer.from_host(np.concatenate(Rs)), adb.DeviceBuffer.from_host(np.concatenate(Ss))
    try:
        adb.batch_set_tuning([0] * 33)
        c, k, _ = adb.batch_join_device(dR.ptr, r_off, dS.ptr, s_off, 0)
    finally:
        adb.batch_set_tuning(None)
        dR.close()
        dS.close()
    for w, (R, S) in enumerate(zip(Rs, Ss)):
        assert (int(c[w]), int(k[w])) == oracle.truth(R, S), sizes[w]
