"""The partitioned joins' device workspace: its size for relations of unlike
sizes, and what a join does where it does not fit.  Free memory is read around
a call and cut down by holding a buffer; counts and checksums are exact."""
import numpy as np
import pytest
import torch

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


def free_bytes():
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def relations():
    kept = []

    def make(n_r, n_s, seed):
        R = adb.gen_pk(n_r, seed)
        S = adb.gen_fk(n_s, R, 0.0, seed + 1)
        kept.extend([adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)])
        return R, S, kept[-2].ptr, kept[-1].ptr

    torch.cuda.empty_cache()
    adb.lib().adb_release_workspace()
    yield make
    for b in kept:
        b.close()
    adb.lib().adb_release_workspace()


@pytest.mark.parametrize("algo", ["PRO", "m-way"])
@pytest.mark.parametrize("n_r,n_s,passes", [
    (4_500_000, 1 << 25, 2),      # a small R, whose partitions ask for two passes over S
    (1 << 25, 20_011, 2),         # an S of less than one CTA's share
    (20_011, 1 << 25, 1),
    (1 << 24, 1 << 24, 2),
])
def test_each_relation_has_its_own_pages(oracle, relations, algo, n_r, n_s, passes):
    R, S, dR, dS = relations(n_r, n_s, 61)
    before = free_bytes()
    got = adb.join_device(algo, dR, n_r, dS, n_s)
    took = before - free_bytes()
    assert (got.count, got.checksum) == oracle.pk_truth(R, S)
    # per pass 8 bytes a tuple in pages, a quarter for partly filled ones and the lists,
    # an eighth that the workspace allocates beyond its need; 64 MiB of fixed tables
    assert took <= passes * 8 * (n_r + n_s) * 1.25 * 1.125 + (64 << 20)


@pytest.mark.parametrize("algo,n_r,n_s,room", [
    ("PRO", 4_500_000, 1 << 26, 900 << 20),       # two passes take 1.2 GB, one 0.6
    ("PRH", 4_500_000, 1 << 26, 900 << 20),
    ("m-way", 4_500_000, 1 << 26, 900 << 20),
    ("NPO", 1 << 25, 1 << 25, 1000 << 20),        # pages 1.15 GB, the one table 0.8
])
def test_a_join_that_does_not_fit_takes_less(oracle, relations, algo, n_r, n_s, room):
    R, S, dR, dS = relations(n_r, n_s, 63)
    want = oracle.pk_truth(R, S)
    usual = adb.join_device(algo, dR, n_r, dS, n_s)
    assert (usual.count, usual.checksum) == want
    adb.lib().adb_release_workspace()
    hold = adb.DeviceBuffer(free_bytes() - room)
    try:
        got = adb.join_device(algo, dR, n_r, dS, n_s)
    finally:
        hold.close()
    assert (got.count, got.checksum) == want
    assert got.kernels < usual.kernels      # one pass instead of two, or NPO's build and probe


def test_a_join_that_fits_in_no_form_is_refused(relations):
    _, _, dR, dS = relations(1 << 24, 1 << 24, 65)
    hold = adb.DeviceBuffer(free_bytes() - (64 << 20))
    try:
        for algo in ("PRO", "NPO", "m-way"):
            with pytest.raises(adb.AdbError) as e:
                adb.join_device(algo, dR, 1 << 24, dS, 1 << 24)
            assert e.value.status == adb.ADB_ERR_OOM
    finally:
        hold.close()
    assert adb.join_device("PRO", dR, 1 << 24, dS, 1 << 24).count == 1 << 24


def test_a_fan_out_of_2_16_is_taken(oracle, relations):
    """Results do not depend on the fan-out; the page set of 2^16 partitions is larger than that of 2^15."""
    R, S, dR, dS = relations(1 << 20, 1 << 20, 67)
    want = oracle.pk_truth(R, S)
    took = []
    for fanout in (1 << 15, 1 << 16, 1 << 20):
        adb.lib().adb_release_workspace()
        before = free_bytes()
        got = adb.join_device("m-way", dR, 1 << 20, dS, 1 << 20, adb.default_params(part_fanout=fanout))
        took.append(before - free_bytes())
        assert (got.count, got.checksum) == want
    assert took[0] < took[1] == took[2]


def fmix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


@pytest.mark.parametrize("n_r", [1 << 31, (1 << 31) + 12345])
def test_npo_of_2_31_build_tuples(relations, n_r):
    """The largest build sides are partitioned like the others (the one table costs a random
    DRAM access per tuple), and none is grouped into regions of more than 2^32 slots."""
    n_s = 3_000_001
    torch.cuda.empty_cache()
    if free_bytes() < 130 << 30:
        pytest.skip("needs 130 GB of free device memory")
    bufs = [adb.DeviceBuffer(8 * n_r), adb.DeviceBuffer(8 * n_s), adb.DeviceBuffer(4 * n_s)]
    dR, dS, dI = (b.ptr for b in bufs)
    try:
        adb._check(adb.lib().adb_gen_pk(dR, n_r, 71, 1))
        adb._check(adb.lib().adb_gen_fk(dS, n_s, dR, n_r, 0.0, 72, dI, 1))
        s = bufs[1].to_host(np.uint64, n_s)
        i = bufs[2].to_host(np.uint32, n_s).astype(np.uint64)     # the R row each S row was drawn from
        key, pay = s >> np.uint64(32), s & np.uint64(0xFFFFFFFF)
        want = int(fmix((key << np.uint64(32) | i) ^ fmix(pay << np.uint64(32) | key)).sum(dtype=np.uint64))
        got = adb.join_device("NPO", dR, n_r, dS, n_s)
        assert (got.count, got.checksum) == (n_s, want) and got.kernels > 4
        for bits in (-1, 3):
            if bits > 0 and n_r == 1 << 31:
                continue                                          # regions of 2^32 slots: as at any size
            got = adb.join_device("NPO", dR, n_r, dS, n_s, adb.default_params(radix_bits=bits))
            assert (got.count, got.checksum) == (n_s, want) and got.kernels == 2
    finally:
        for b in bufs:
            b.close()
