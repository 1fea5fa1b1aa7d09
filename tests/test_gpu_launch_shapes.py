"""The shapes of the worklist launches, as the CUDA profiler records them, and the bits of both register caps."""
import json

import numpy as np
import pytest

import soundings

pytestmark = pytest.mark.gpu

LIST1 = "uwshcu_fp64_kernel<%d, 5, 3, 0"


def _launches(torch, fn, tmp_path):
    """(name, blocks, microseconds) of every kernel that fn launches."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    p.export_chrome_trace(path)
    got = [(e["name"], e["args"]["grid"][0], e["dur"]) for e in json.load(open(path))["traceEvents"]
           if e.get("cat") == "kernel"]
    if not got:
        pytest.skip("the CUDA profiler records nothing here")
    return got


def test_streams_of_the_past_do_not_narrow_a_call(uw, cuda, tmp_path):
    """256 columns on one stream: a block of four warps for every four of them, also in a process that has
    run on 32 streams before, once 32 calls lie behind."""
    torch = cuda
    assert uw.init_default() == 0
    assert uw.set_precision(uw.PREC_FP64) == 0
    c = uw.DeviceCase(soundings.make_soundings(256, 30, seed=41))

    def call(stream=None):
        c.reset_cush()
        assert c.launch(stream=stream) == 0, uw.last_cuda_error()

    call()
    for _ in range(32):
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        call(s)
        torch.cuda.current_stream().wait_stream(s)
    for _ in range(40):
        call()
    torch.cuda.synchronize()
    grids = [g for name, g, _ in _launches(torch, call, tmp_path) if LIST1 % 32 in name]
    assert grids == [64], grids


LONG_US, EMPTY_US = 1000.0, 200.0   # a launch that does the work takes milliseconds, one that returns at once microseconds


def _repeated(s, times):
    """The sounding's columns `times` over."""
    n = s["ncol"]
    out = {k: np.tile(v, (1,) * (v.ndim - 1) + (times,)) if isinstance(v, np.ndarray) and v.shape[-1:] == (n,)
           else v for k, v in s.items()}
    out["ncol"] = n * times
    return out


def _same_bits(got, want, times):
    return [k for k in want if not np.array_equal(got[k].reshape(got[k].shape[:-1] + (times, -1)),
                                                  np.broadcast_to(want[k][..., None, :], want[k].shape[:-1] + (times, want[k].shape[-1])))]


def _single_pass(uw, s):
    assert uw.set_schedule(uw.SCHED_SINGLE_PASS) == 0
    try:
        c = uw.DeviceCase(s)
        assert c.launch() == 0 and c.status() == 0, uw.last_cuda_error()
        return c.outputs_numpy()
    finally:
        assert uw.set_schedule(uw.SCHED_DEFAULT) == 0


def _worked(launches, stem, short, dense):
    """Whether the instantiation `dense` of a kernel did the work; the other one is absent or returned at once."""
    us = {tag: max([d for name, _, d in launches if stem + tag in name], default=0.0) for tag in (short, dense)}
    assert max(us.values()) > LONG_US and min(us.values()) < EMPTY_US, us
    return us[dense] > us[short]


@pytest.mark.parametrize("levels,kp,rh,times,slots", [
    (30, 32, (0.55, 0.76), 49, 0),   # many columns, few of which convect
    (30, 32, (0.75, 0.97), 20, 0),   # fewer columns, a longer worklist
    (30, 32, (0.75, 0.97), 20, 5000),   # and not enough hand-off slots
    (51, 64, (0.75, 0.97), 24, 0),
    (51, 64, (0.55, 0.76), 24, 0),
])
def test_the_worklist_decides_the_register_cap(uw, cuda, tmp_path, levels, kp, rh, times, slots):
    assert uw.init_default() == 0
    assert uw.set_precision(uw.PREC_FP64) == 0
    assert uw.set_hand_slots(slots) == 0
    try:
        _check_register_cap(uw, cuda, tmp_path, levels, kp, rh, times)
    finally:
        assert uw.set_hand_slots(0) == 0


def _check_register_cap(uw, cuda, tmp_path, levels, kp, rh, times):
    base = soundings.make_soundings(7001, levels, seed=levels, rh_pbl=rh)
    want = _single_pass(uw, base)
    c = uw.DeviceCase(_repeated(base, times))
    assert uw.set_profiling(1) == 0
    uw.profile_read()
    assert c.launch() == 0 and c.status() == 0, uw.last_cuda_error()
    n = uw.profile_read()[3]
    assert uw.set_profiling(0) == 0

    def call():
        c.reset_cush()
        assert c.launch() == 0, uw.last_cuda_error()

    launches = _launches(cuda, call, tmp_path)
    dense = n > 4 * 128 * cuda.cuda.get_device_properties(0).multi_processor_count
    for mode in (3, 4):
        assert _worked(launches, "uwshcu_fp64_kernel<%d, 5, %d, 0, " % (kp, mode), "0>", "1>") == dense, n
    assert not _same_bits(c.outputs_numpy(), want, times)


@pytest.mark.parametrize("rh,times", [((0.55, 0.76), 22), ((0.75, 0.97), 22)])
def test_a_batch_decides_by_its_class(uw, cuda, tmp_path, rh, times):
    assert uw.init_default() == 0
    assert uw.set_precision(uw.PREC_FP64) == 0
    bases = [soundings.make_soundings(7001, levels, seed=60 + levels, rh_pbl=rh) for levels in (30, 51)]
    wants = [_single_pass(uw, b) for b in bases]
    cases = [uw.DeviceCase(_repeated(b, times)) for b in bases]
    plan = uw.BatchPlan(cases)
    try:
        def call():
            for c in cases:
                c.reset_cush()
            assert plan.run() == 0, uw.last_cuda_error()

        call()
        launches = _launches(cuda, call, tmp_path)
        assert plan.status() == 0
        for kp in (32, 64):
            moist = rh[0] > 0.7
            assert _worked(launches, "uwshcu_batch_list<%d, 5, " % kp, "4, 0, 3>", "7, 0, 3>") == moist
            assert _worked(launches, "uwshcu_batch_resume<%d, 5, 0, " % kp, "5>", "7>") == moist
    finally:
        plan.close()
    for c, want in zip(cases, wants):
        assert not _same_bits(c.outputs_numpy(), want, times)
