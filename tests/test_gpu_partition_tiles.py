"""Partition passes at the edges of their tiles: CTA chunks and work units
around 6144 and 8192 tuples, one pass and two, an input that is not 16-byte
aligned, one side much larger than the other, a digit that holds most of every
tile; batched windows around one tile.  Whole numbers: exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def rel(n, kind, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << 22, size=n, dtype=np.uint64).astype(np.uint32)
    if kind == "hot":
        k[rng.random(n) < 0.7] = 0x155555
    return adb.tuples(k)


def join_at(algo, R, S, par, skip):
    """The join of R[skip:] and S[skip:], from device pointers 8 * skip bytes into their buffers."""
    dR, dS = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)
    try:
        o = adb.join_device(algo, dR.ptr + 8 * skip, len(R) - skip, dS.ptr + 8 * skip, len(S) - skip, par)
        return o.count, o.checksum
    finally:
        dR.close()
        dS.close()


@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("fanout", [2, 64, 512, 1024, 1 << 14])
@pytest.mark.parametrize("n", [1, 6143, 6145, 8191, 8192, 8193, 148 * 6144 + 1, 148 * 8192 + 1])
def test_tile_edges(oracle, n, fanout, skip):
    R, S = rel(3000 + skip, "spread", 1), rel(n + skip, "spread", n)
    par = adb.default_params(part_fanout=fanout)
    assert join_at("m-way", R, S, par, skip) == oracle.truth(R[skip:], S[skip:])
    assert join_at("m-way", S, R, par, skip) == oracle.truth(S[skip:], R[skip:])


@pytest.mark.parametrize("algo,bits", [("PRO", 1), ("PRO", 6), ("PRO", 9), ("PRO", 14), ("m-way", 6), ("m-way", 14)])
@pytest.mark.parametrize("n", [20000, 3 * 148 * 8192 + 77])
def test_hot_digit(oracle, algo, bits, n):
    R, S = rel(4000, "spread", 2), rel(n, "hot", 3)
    par = adb.default_params(radix_bits=bits) if algo == "PRO" else adb.default_params(part_fanout=1 << bits)
    assert join_at(algo, R, S, par, 0) == oracle.truth(R, S)


def test_batch_windows_around_a_tile(oracle):
    sizes = [1, 4097, 8191, 8192, 8193, 16383, 16385, 131071, 131073]
    Rs = [rel(n, "spread", n) for n in sizes]
    Ss = [rel(n, "hot" if i & 1 else "spread", 7 * n) for i, n in enumerate(reversed(sizes))]
    r_off = np.concatenate([[0], np.cumsum([len(r) for r in Rs])]).astype(np.uint64)
    s_off = np.concatenate([[0], np.cumsum([len(s) for s in Ss])]).astype(np.uint64)
    dR, dS = adb.DeviceBuffer.from_host(np.concatenate(Rs)), adb.DeviceBuffer.from_host(np.concatenate(Ss))
    c, k, _ = adb.batch_join_device(dR.ptr, r_off, dS.ptr, s_off)
    dR.close()
    dS.close()
    for w, (R, S) in enumerate(zip(Rs, Ss)):
        assert (int(c[w]), int(k[w])) == oracle.truth(R, S), w
