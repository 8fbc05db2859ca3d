"""PMJ's merges and merge joins at the edges of their 2048-tuple tiles and of
the 8192-tuple sorted blocks: sizes around both, runs of equal keys longer than
a tile, one side empty before the other, the largest key.  Whole numbers: exact."""
import numpy as np
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def rel(n, kind, seed):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    if kind == "few":
        k = k % np.uint32(max(n // 1000, 2))          # runs of about 1000
    elif kind == "runs":
        k[rng.random(n) < 0.3] = 0xFFFFFFFF           # one run over several tiles
    elif kind == "apart":
        k = (k >> np.uint32(1)) | np.uint32((seed & 1) << 31)   # all of R below all of S
    return adb.tuples(k)


@pytest.mark.parametrize("kind", ["spread", "few", "runs", "apart"])
@pytest.mark.parametrize("nr,ns", [(1, 1), (1, 2048), (2047, 1), (1024, 1024), (2048, 2049), (8191, 8193), (8192, 8192),
                                   (16385, 2047), (24577, 33), (70001, 5000)])
def test_sizes(oracle, kind, nr, ns):
    R, S = rel(nr, kind, 2 * nr), rel(ns, kind, 2 * ns + 1)
    S["key"][: min(nr, ns) // 2] = R["key"][: min(nr, ns) // 2]
    for algo, par in (("PMJ_JM_NP", adb.default_params()), ("PMJ_JM_NP", adb.default_params(progressive_step=3))):
        got = adb.join(algo, R, S, par)
        assert (got.count, got.checksum) == oracle.truth(R, S)
