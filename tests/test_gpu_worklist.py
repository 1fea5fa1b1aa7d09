"""The worklist that the trigger pass's keys give (ordered by release level in tiles of 8,192 columns) and
its spreading over warps: every column that convects is on it exactly once, at the edges of warps, tiles
and spreading (one column to a warp up to 592 of them, 32 from 9,473 on).  The single-pass schedule, which
uses no worklist, computes the same bits; so must the two worklist schedules, from device arrays and
through the chunked host entry, and the tangent-linear model's values."""
import numpy as np
import pytest

import soundings

pytestmark = pytest.mark.gpu


def _differ(a, b):
    return [k for k in a if not np.array_equal(a[k], b[k])]


@pytest.mark.parametrize("ncol,rh", [
    (1, (0.90, 0.97)), (31, (0.90, 0.97)), (33, (0.60, 0.95)), (593, (0.97, 0.99)), (1300, (0.60, 0.95)),
    (8191, (0.60, 0.95)), (8192, (0.97, 0.99)), (8193, (0.55, 0.76)), (24577, (0.70, 0.95)), (500, (0.05, 0.10)),
])
def test_worklist_holds_every_convecting_column_once(uw, cuda, ncol, rh):
    assert uw.init_default() == 0
    assert uw.set_precision(uw.PREC_FP64) == 0
    s = soundings.make_soundings(ncol, 30, seed=700 + ncol, rh_pbl=rh)
    try:
        assert uw.set_schedule(uw.SCHED_SINGLE_PASS) == 0
        c = uw.DeviceCase(s, diag=True)
        assert c.launch_member() == 0 and c.status() == 0, uw.last_cuda_error()
        want = c.outputs_numpy()
        for sched in (uw.SCHED_SORTED, uw.SCHED_TWO_PHASE):
            assert uw.set_schedule(sched) == 0
            c = uw.DeviceCase(s, diag=True)
            for v in c.out.values():
                v.fill_(-777.0)
            c.reset_cush()
            assert c.launch_member() == 0 and c.status() == 0, uw.last_cuda_error()
            got = c.outputs_numpy()
            assert not _differ(got, want), (sched, _differ(got, want))
        assert uw.set_schedule(uw.SCHED_SORTED) == 0
        assert uw.set_pipeline(3000, 3) == 0
        rc, host = uw.compute_host(s)
        assert rc == 0, uw.last_cuda_error()
        assert not [k for k in host if not np.array_equal(host[k], want[k])]
        c = uw.DeviceCase(s)
        uw.tangent_launch(c, {"t0": c.inp["t0"] * 1.0e-3})
        assert c.status() == 0
        got = c.outputs_numpy()
        assert not [k for k in got if not np.array_equal(got[k], want[k])]
    finally:
        assert uw.set_pipeline(-1, 0) == 0
        assert uw.set_schedule(uw.SCHED_DEFAULT) == 0
