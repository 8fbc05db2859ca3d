"""Which form NPO's dispatch takes for a large S, seen by the launches of the
call (two for the table), on both sides of each line; exact either way."""
import pytest

import alliancedb_b200 as adb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_r,n_s,table", [
    (7 << 19, 1 << 16, True), ((7 << 19) + 1, 1 << 16, False),
    (1 << 22, 1 << 23, True), (1 << 22, (1 << 23) - 1, False), ((1 << 22) + 1, 1 << 23, False),
    ((1 << 22) + 1, 8 * ((1 << 22) + 1), True), ((1 << 22) + 1, 8 * ((1 << 22) + 1) - 1, False),
    (7 << 20, 56 << 20, True), ((7 << 20) + 1, (56 << 20) + 8, False),
])
def test_route(n_r, n_s, table):
    dR, dS = adb.DeviceBuffer(8 * n_r), adb.DeviceBuffer(8 * n_s)
    try:
        adb._check(adb.lib().adb_gen_pk(dR.ptr, n_r, 5, 1))
        adb._check(adb.lib().adb_gen_fk(dS.ptr, n_s, dR.ptr, n_r, 1.0, 6, None, 1))
        got = adb.join_device("NPO", dR.ptr, n_r, dS.ptr, n_s)
        other = adb.join_device("PRO", dR.ptr, n_r, dS.ptr, n_s)
        assert (got.kernels == 2) == table
        assert got.count == n_s and (got.count, got.checksum) == (other.count, other.checksum)
    finally:
        dR.close()
        dS.close()
