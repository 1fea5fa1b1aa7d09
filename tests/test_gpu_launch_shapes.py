"""The shapes of the worklist launches, as the CUDA profiler records them."""
import json

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
