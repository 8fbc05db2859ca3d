"""A call that failed half-way leaves nothing behind: the next one, on another
stream, must not share its accumulators or workspace with kernels that the
failed call had queued, nor have its sums cleared by that call's clean-up.
ADB_TEST_CALL_FAILS makes the host give up with the kernels queued; counts and
checksums are exact."""
import pytest
import torch

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu

ADB_TEST_CALL_FAILS = 2


def on_device(n_r, n_s, seed):
    R = adb.gen_pk(n_r, seed)
    S = adb.gen_fk(n_s, R, 0.0, seed + 1)
    return R, S, adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)


@pytest.mark.parametrize("algo,n", [("PRO", 1 << 24), ("NPO", 1 << 21), ("m-way", 1 << 22), ("PRH", 1 << 13)])
def test_next_call_on_another_stream(oracle, algo, n):
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    R, S, dR, dS = on_device(n, n, 41)
    r, s, dr, ds = on_device(3000, 70001, 43)
    want = oracle.pk_truth(R, S), oracle.pk_truth(r, s)
    fails = adb.default_params(test_flags=ADB_TEST_CALL_FAILS)
    for _ in range(20):
        with pytest.raises(adb.AdbError) as e:
            adb.join_device(algo, dR.ptr, n, dS.ptr, n, fails, stream=a)
        assert e.value.status == adb.ADB_ERR_DEVICE
        got = adb.join_device(algo, dr.ptr, 3000, ds.ptr, 70001, stream=b)
        assert (got.count, got.checksum) == want[1]
        got = adb.join_device(algo, dR.ptr, n, dS.ptr, n, stream=b)
        assert (got.count, got.checksum) == want[0]


def test_an_error_is_reported_once(oracle):
    """A CUDA call's error belongs to the call that made it, not to the next launch."""
    R = adb.gen_pk(3000, 45)
    S = adb.gen_fk(5000, R, 0.0, 46)
    dR, dS = adb.DeviceBuffer.from_host(R), adb.DeviceBuffer.from_host(S)
    assert adb.lib().adb_host_free_pinned(R.ctypes.data) == adb.ADB_ERR_DEVICE   # not pinned memory
    got = adb.join_device("PRO", dR.ptr, 3000, dS.ptr, 5000)
    assert (got.count, got.checksum) == oracle.truth(R, S)


@pytest.mark.parametrize("algo", ["PRO", "NPO", "m-way", "SHJ_JM_NP"])
@pytest.mark.parametrize("word,says", [(2, "table full"), (3, "page pool")])
def test_a_kernels_check_is_not_a_timeout(oracle, algo, word, says):
    R = adb.gen_pk(20000, 47)
    S = adb.gen_fk(30000, R, 0.0, 48)
    with pytest.raises(adb.AdbError) as e:
        adb.join(algo, R, S, adb.default_params(test_flags=word << 8))
    assert e.value.status == adb.ADB_ERR_DEVICE and says in str(e.value)
    got = adb.join(algo, R, S)
    assert (got.count, got.checksum) == oracle.pk_truth(R, S)


@pytest.mark.parametrize("n", [1 << 14, (7 << 19) + 1])
def test_npo_has_no_wait_to_run_out_at_any_size(oracle, n):
    R = adb.gen_pk(n, 49)
    S = adb.gen_fk(n, R, 0.0, 50)
    got = adb.join("NPO", R, S, adb.default_params(test_flags=1))
    assert (got.count, got.checksum) == oracle.pk_truth(R, S)
