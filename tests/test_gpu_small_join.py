"""The single-launch hash join of a small build side: chunk edges of R, ragged
S shares, repeated keys, extreme keys, materialisation, and the sizes either
side of its dispatch rule.  Whole numbers: exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def rel(n, space, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, space, size=n, dtype=np.uint64).astype(np.uint32)
    k[: min(3, n)] = np.array([0, 0xFFFFFFFF, 0x80000000], np.uint32)[: min(3, n)]
    return adb.tuples(k, rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32))


@pytest.mark.parametrize("algo", ["PRO", "NPO"])
@pytest.mark.parametrize("n_r,n_s", [(1, 1), (2, 127), (3, 128), (5, 2049), (4095, 129), (8191, 2047), (8192, 2048),
                                     (8193, 5000), (16384, 301), (16385, 300), (30000, 606211), (1 << 18, 32),
                                     (1 << 18, 33), (40000, 1 << 20), (1 << 20, 65), (7, 1 << 20)])
@pytest.mark.parametrize("space", [1 << 32, 3000])
def test_sizes(oracle, algo, n_r, n_s, space):
    if space == 3000 and n_r * n_s > 1 << 32:
        space = 1 << 17
    R, S = rel(n_r, space, n_r), rel(n_s, space, n_s + 1)
    got = adb.join(algo, R, S)
    assert (got.count, got.checksum) == oracle.truth(R, S)


def test_low_bits_equal(oracle):
    # keys that differ only above bit 18
    k = (np.arange(8192, dtype=np.uint32) << np.uint32(19)) | np.uint32(5)
    R, S = adb.tuples(k), adb.tuples(np.tile(k, 3))
    got = adb.join("PRO", R, S)
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("n_r", [100, 8192, 20000])
def test_materialise_and_calls_in_a_row(oracle, n_r):
    R, S = rel(n_r, 5000, 3), rel(3001, 5000, 4)
    want = oracle.truth(R, S)
    dR, dS = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)
    for cap in (want[0], want[0] // 2):
        out = adb.DeviceBuffer(8 * max(cap, 1))
        for _ in range(2):   # the accumulators are back at zero after each call
            got = adb.join_materialize_device("NPO", dR.ptr, n_r, dS.ptr, 3001, out.ptr, cap)
            assert (got.count, got.checksum) == want and got.materialized == cap
        rows = out.to_host(np.uint64, cap)
        keys, n = np.unique(S.view(np.uint64), return_counts=True)
        per_key = dict(zip(*np.unique(R["key"], return_counts=True)))
        have, m = np.unique(rows, return_counts=True)
        full = {int(w): int(c) * int(per_key.get(np.uint32(w >> np.uint64(32)), 0)) for w, c in zip(keys, n)}
        assert all(c <= full[int(w)] for w, c in zip(have, m))
        if cap == want[0]:
            assert sum(full.values()) == cap and all(c == full[int(w)] for w, c in zip(have, m))
        out.close()
    dR.close()
    dS.close()


def test_unaligned_relations(oracle):
    R, S = rel(1001, 2000, 8), rel(4099, 2000, 9)
    dR, dS = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)
    got = adb.join_device("PRO", dR.ptr + 8, 1000, dS.ptr + 8, 4098)
    assert (got.count, got.checksum) == oracle.truth(R[1:], S[1:])
    dR.close()
    dS.close()
