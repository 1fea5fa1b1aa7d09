"""The FP64 saturation adjustment (conden_f64, whose divisions go by uw_rcp) against the general one (conden, which it
falls back to), compiled from the kernels' own header: every bit of every result, at the edges of the
saturation table and of its range, at divisors that uw_rcp_ok refuses, and far outside the atmosphere.
Beside it the parts: uw_quotient, and the hardware's approximation that uw_rcp starts from."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import soundings

pytestmark = pytest.mark.gpu

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-and-climate-model_b200")

SOURCE = """
#include "uwshcu_fp64_kernel.cuh"
#include <cstring>

namespace {
__global__ void conden_kernel(const double* in, double* general, double* fast, int n)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double p = in[i], ex = in[n + i], thl = in[2 * n + i], qt = in[3 * n + i];
    for (int f = 0; f < 2; f++) {
        const CondenOut r = f ? conden_f64(p, ex, thl, qt, tbl) : conden_any(p, ex, thl, qt, tbl);
        double* o = (f ? fast : general) + i;
        o[0] = r.th;
        o[n] = r.qv;
        o[2 * n] = r.ql;
        o[3 * n] = r.qi;
        o[4 * n] = r.rv0;
        o[5 * n] = r.id;
    }
}
__global__ void quotient_kernel(const double* a, const double* b, double* got, double* want, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const UwQuotient r = uw_quotient(a[i], b[i]);
    const double q = a[i] / b[i];
    got[i] = r.q, got[n + i] = r.y, got[2 * n + i] = r.z;
    want[i] = q, want[n + i] = 1.0 / b[i], want[2 * n + i] = -q / b[i];
}
// residuals 1 - b y of the approximation at b in [1, 2): the 20 upper bits of the fraction from the thread, `low` below
__global__ void approx_kernel(unsigned low, double* residual)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double b = __hiloint2double(0x3ff00000 | i, (int)low);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    residual[i] = fma(-b, y, 1.0);
}
int high_word(double x)
{
    long long b;
    std::memcpy(&b, &x, sizeof(b));
    return (int)(b >> 32);
}
}  // namespace

extern "C" int set_constants(double xlv, double xlf, double cp, double r, double ep2, double tmin, double tmax,
                             double epsqs, const double* table)
{
    UwConst k{};
    k.xlv = xlv, k.xls = xlv + xlf, k.cp = cp, k.r = r, k.ep2 = ep2, k.tmin = tmin, k.tmax = tmax, k.epsqs = epsqs;
    k.rinv = 1.0 / r, k.cpinv = 1.0 / cp, k.omeps = 1.0 - epsqs;
    k.tlo = high_word(tmin) + 1, k.tnum = high_word(tmax) - k.tlo;
    cudaError_t e = cudaMemcpyToSymbol(c, &k, sizeof(k));
    return e != cudaSuccess ? e : cudaMemcpyToSymbol(c_estbl, table, sizeof(double) * UW_TBL);
}
extern "C" int run_conden(const double* in, double* general, double* fast, int n)
{
    conden_kernel<<<(n + 127) / 128, 128>>>(in, general, fast, n);
    return cudaDeviceSynchronize();
}
extern "C" int run_quotient(const double* a, const double* b, double* got, double* want, int n)
{
    quotient_kernel<<<(n + 127) / 128, 128>>>(a, b, got, want, n);
    return cudaDeviceSynchronize();
}
extern "C" int run_approx(unsigned low, double* residual)
{
    approx_kernel<<<(1 << 20) / 128, 128>>>(low, residual);
    return cudaDeviceSynchronize();
}
"""

TMIN, TMAX = 173.16, 375.16


@pytest.fixture(scope="module")
def lib(uw, cuda, tmp_path_factory):
    sys.path.insert(0, PKG)
    import build
    d = tmp_path_factory.mktemp("conden")
    src, so = d / "conden.cu", d / "conden.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc()] + build.ARCH + build.COMMON + ["-fmad=false", "-shared", str(src), "-o", str(so)], check=True)
    L = ctypes.CDLL(str(so))
    f = ctypes.c_double
    s = soundings
    table = uw.estbl()
    assert L.set_constants(f(s.LATVAP), f(s.LATICE), f(s.CPAIR), f(s.RAIR), f(s.EPSILO), f(TMIN), f(TMAX), f(s.EPSILO),
                           table.ctypes.data_as(ctypes.c_void_p)) == 0
    L.torch, L.table = cuda, table
    return L


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _conden(lib, p, ex, thl, qt):
    torch = lib.torch
    n = len(p)
    x = torch.from_numpy(np.stack([np.asarray(a, dtype=np.float64) for a in (p, ex, thl, qt)])).cuda()
    general, fast = (torch.full((6, n), -7.0, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    assert lib.run_conden(_ptr(x), _ptr(general), _ptr(fast), n) == 0
    return general.cpu().numpy(), fast.cpu().numpy()


def _differing(a, b):
    nan = np.isnan(a)
    return np.flatnonzero(((nan != np.isnan(b)) | (~nan & (a.view(np.int64) != b.view(np.int64)))).reshape(-1, a.shape[-1]).any(axis=0))


def _refused(b):
    """The doubles that uw_rcp_ok refuses."""
    with np.errstate(invalid="ignore"):
        return ~((b >= 2.0 ** -100) & (b < 2.0 ** 100)) | ((b.view(np.uint64) & np.uint64(0xffffffff)) == 0xffffffff)


def _same(lib, p, ex, thl, qt):
    general, fast = _conden(lib, p, ex, thl, qt)
    bad = _differing(general, fast)
    assert bad.size == 0, [(p[i], ex[i], thl[i], qt[i], general[:, i], fast[:, i]) for i in bad[:3]]
    return general


def _neighbours(x):
    return [np.nextafter(x, -np.inf), x, np.nextafter(x, np.inf)]


def test_atmosphere(lib):
    """The atmosphere, and a humidity at which the first look-up of the saturation decides by its last bit."""
    rng = np.random.default_rng(0)
    n = 2_000_000
    p = rng.uniform(5.0e3, 1.05e5, n)
    ex = (p / 1.0e5) ** 0.2857
    thl = rng.uniform(170.0, 330.0, n) / ex
    qt = 10.0 ** rng.uniform(-9, -1, n)
    general = _same(lib, p, ex, thl, qt)
    assert general[1].min() >= 0.0 and (general[2] > 0.0).sum() > 10_000
    for q in (general[4], np.nextafter(general[4], 0.0), np.nextafter(general[4], 1.0)):
        _same(lib, p, ex, thl, q)


def test_edges_of_the_table_and_of_the_range(lib):
    """Temperatures at, below and above every step of the table and both its ends; divisors at and beside the
    refused ones; values that no atmosphere has."""
    lows = np.array([0xffffffff, 0xfffffffe, 0], dtype=np.uint64)
    steps = TMIN + np.arange(0, 203)
    t = [x for s in steps for x in _neighbours(s)]
    for e in (TMIN, TMAX):                # the words beside those of the ends decide whether a temperature is clamped
        high = int(np.float64(e).view(np.uint64)) >> 32
        for h in (high - 1, high, high + 1):
            t += list((np.uint64(h << 32) | lows).view(np.float64))
    hot = (np.array([250.0, 300.0, 180.0]).view(np.uint64) & ~np.uint64(0xffffffff))
    t += [x for h in hot for x in (h | lows).view(np.float64)]
    t += [0.0, -0.0, -1.0, -250.0, 1.0e-40, 1.0e-300, 5e-324, 1.0, 1.0e3, 1.0e10, 1.0e31, 1.0e300, 1.7e308, -1.0e300,
          np.inf, -np.inf, np.nan]
    t = np.array(t)
    p = np.array([1.0e5, 5.0e4, 1.0e3, 10.0, 1.0, 1.0e-3, 0.0, -1.0, -1.0e5, 1.0e31, 1.0e300, np.inf, np.nan])
    q = np.array([0.0, -0.0, 1.0e-12, 1.0e-3, 2.0e-2, 0.5, 1.0, 2.0, -1.0e-3, 1.0e10, 1.0e300, 1.7e308, 5e-324, np.inf, np.nan])
    P, T, Q = (a.ravel() for a in np.meshgrid(p, t, q, indexing="ij"))
    assert _refused(T).sum() > 1000      # the Newton steps start at the divisor T
    _same(lib, P, np.ones_like(P), T, Q)


def test_a_refused_saturation_divisor(lib):
    """p - (1 - eps) es(T) with the refused low word, zero and negative: the whole call goes the general way."""
    omeps = 1.0 - soundings.EPSILO
    n = np.arange(5, 195)
    es = lib.table[n]                     # at T = tmin + n the table's value itself, if the sum is exact
    T = TMIN + n
    exact = (T - TMIN) == n
    T, es = T[exact], es[exact]
    assert len(T) > 50
    d0 = ((np.float64(7.0e4).view(np.uint64) & ~np.uint64(0xffffffff)) | np.uint64(0xffffffff)).view(np.float64)
    p = d0 + omeps * es
    for _ in range(4):                    # the last bit of p that gives d0
        p = np.where(p - omeps * es < d0, np.nextafter(p, np.inf), np.where(p - omeps * es > d0, np.nextafter(p, 0.0), p))
    hit = p - omeps * es == d0
    assert hit.sum() > 20
    sets = [(p[hit], T[hit]), (omeps * es, T), (np.nextafter(omeps * es, 0.0), T), (0.5 * omeps * es, T)]
    P, TT = (np.concatenate(x) for x in zip(*sets))
    for qt in (0.0, 1.0e-4, 2.0e-2, 0.9, 1.5):
        _same(lib, P, np.ones_like(P), TT, np.full_like(P, qt))


def test_quotient_and_its_partials(lib):
    torch = lib.torch
    rng = np.random.default_rng(5)
    n = 1_000_000
    a = rng.standard_normal(n) * 2.0 ** rng.uniform(-500, 500, n)
    b = rng.standard_normal(n) * 2.0 ** rng.uniform(-500, 500, n)
    special = np.array([0.0, -0.0, 1.0, -3.0, 5e-324, np.inf, -np.inf, np.nan, 2.0 ** -1022, 1.7e308, 2.0 - 2.0 ** -52])
    a[: len(special) ** 2] = np.repeat(special, len(special))
    b[: len(special) ** 2] = np.tile(special, len(special))
    A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    got, want = (torch.empty((3, n), dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    assert lib.run_quotient(_ptr(A), _ptr(B), _ptr(got), _ptr(want), n) == 0
    bad = _differing(got.cpu().numpy(), want.cpu().numpy())
    assert bad.size == 0, [(a[i], b[i]) for i in bad[:3]]


@pytest.mark.parametrize("low", [0, 1, 0x7fffffff, 0x80000000, 0xffffffff])
def test_the_approximation_is_close_enough(lib, low):
    """Every upper half of a significand: the residual below 2^-18, with which the cubic step of uw_rcp leaves 2^-54."""
    torch = lib.torch
    res = torch.empty(1 << 20, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_approx(ctypes.c_uint(low), _ptr(res)) == 0
    assert res.abs().max().item() < 2.0 ** -18
