"""The rules that size the worklist launches (csrc/uw_schedule.h), compiled for the CPU: every entry of a
worklist is handed to exactly one thread of the grid that the host launches, whatever its length turns out
to be, at the true edges of the spreading; and the streams a call shares the GPU with are those in use."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-and-climate-model_b200", "csrc")

SHIM = """
#include "uw_schedule.h"
// the threads of a launch over `n` entries at most that get one of the `count` entries; 0 if an entry is missing,
// taken twice or out of range
extern "C" int covered(int n, int count, int spread, int block, unsigned char* taken)
{
    const int threads = (uw_list_threads(n, spread) + block - 1) / block * block;
    int got = 0;
    for (int t = 0; t < threads; t++) {
        const int e = uw_spread(count, spread, t);
        if (e < 0) continue;
        if (e >= count || taken[e]) return -1;
        taken[e] = 1;
        got++;
    }
    return got;
}
extern "C" int lanes(int count, int spread)
{
    int n = 0;
    for (int t = 0; t < 32; t++) n += uw_spread(count, spread, t) >= 0;
    return n;
}
extern "C" int shares(unsigned long long last, unsigned long long tick) { return uw_stream_shares(last, tick); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, so = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.shares.argtypes = [ctypes.c_ulonglong] * 2
    return lib


@pytest.mark.parametrize("spread", [0, 1, 18, 74, 148, 592])
@pytest.mark.parametrize("block", [32, 64, 128])
def test_every_entry_has_one_thread(rules, spread, block):
    edges = {0, 1, 2, 31, 32, 33, 127, 128, 129, 1000}
    for lanes in (1, 2, 4, 8, 16, 32):
        edges |= {max(0, spread * lanes + d) for d in (-1, 0, 1)}
    for n in sorted(edges):
        for count in sorted(c for c in edges if c <= n):
            taken = np.zeros(max(count, 1), np.uint8)
            got = rules.covered(n, count, spread, block, taken.ctypes.data_as(ctypes.c_void_p))
            assert got == count and taken[:count].all(), (n, count, spread, block)


def test_a_short_worklist_is_spread(rules):
    for count, want in ((1, 1), (592, 1), (593, 2), (1184, 2), (1185, 4), (9472, 16), (9473, 32), (100000, 32)):
        assert rules.lanes(count, 592) == want, count
    assert rules.lanes(592, 0) == 32


def _sharers(rules, calls):
    """Streams counted at the last of `calls` (a stream each), as the host counts them."""
    last = {}
    for tick, stream in enumerate(calls, 1):
        last[stream] = tick
    return sum(rules.shares(t, len(calls)) for t in last.values())


def test_only_streams_in_use_share(rules):
    assert _sharers(rules, [7]) == 1
    for m in (1, 2, 3, 8, 31, 32):
        assert _sharers(rules, list(range(m)) * 5) == m            # used in turn
    assert _sharers(rules, list(range(32)) + [0] * 32) == 1        # left long ago
    assert _sharers(rules, list(range(8)) + [100] * 32) == 1
    assert _sharers(rules, list(range(32)) + [0] * 10) == 23       # 22 of the latest 32 calls on others
