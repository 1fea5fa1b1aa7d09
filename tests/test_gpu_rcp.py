"""The reciprocal of the FP64 saturation adjustment (uw_rcp, compiled from uw_math.h by itself)
and the divisions built on it (uw_div_by, uw_quot) against the GPU's IEEE division: every bit, over the whole range
that uw_rcp_ok admits, with the significands at which the method is delicate (all ones, which it refuses, one,
their neighbours); and uw_rcp_ok at the ends of that range."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-and-climate-model_b200", "csrc")


def _function(text, head):
    i = text.index(head)
    return re.sub(r"__forceinline__|UW_HD", "inline", text[i: text.index("\n}\n", i) + 3])


@pytest.fixture(scope="module")
def kernels(cuda):
    torch = cuda
    math = open(os.path.join(CSRC, "uw_math.h")).read()
    src = ("#define UW_MUL(a, b) __dmul_rn((a), (b))\n#define HUGE_VAL __longlong_as_double(0x7ff0000000000000ll)\n"
           + _function(math, "static __device__ __noinline__ double uw_div_ieee(")
           + "".join(_function(math, "static __device__ __forceinline__ " + f) for f in (
               "double uw_rcp(", "bool uw_rcp_ok(", "double uw_quot("))
           + "__device__ " + _function(math, "UW_HD double uw_div_by(")
           + """
extern "C" __global__ void rcp_kernel(const double* a, const double* b, double* y, double* q, int* ok, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = uw_rcp(b[i]);
    q[i] = uw_div_by(a[i], b[i], y[i]);
    ok[i] = uw_rcp_ok(b[i]);
}
extern "C" __global__ void quot_kernel(const double* a, const double* b, const double* y, double* q, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = uw_quot(a[i], b[i], y[i]);
}
""")
    k, kq = (torch.cuda._compile_kernel(src, name) for name in ("rcp_kernel", "quot_kernel"))

    def run(a, b):
        a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        y, q = torch.empty_like(b), torch.empty_like(b)
        ok = torch.empty(b.shape, dtype=torch.int32, device="cuda")
        n = b.numel()
        k(grid=((n + 255) // 256, 1, 1), block=(256, 1, 1), args=(a, b, y, q, ok, n))
        return [t.cpu().numpy() for t in (y, q, ok, 1.0 / b, a / b)]

    def quot(a, b):
        a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        q, n = torch.empty_like(b), b.numel()
        kq(grid=((n + 255) // 256, 1, 1), block=(256, 1, 1), args=(a, b, 1.0 / b, q, n))
        return q.cpu().numpy(), (a / b).cpu().numpy()
    run.quot = quot
    return run


@pytest.mark.parametrize("seed", [0, 1])
def test_reciprocal_and_quotient_are_ieee(kernels, seed):
    rng = np.random.default_rng(seed)
    n = 4_000_000
    frac = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    edge = np.array([0, 1, 2, (1 << 52) - 1, (1 << 52) - 2, (1 << 52) - 3, 1 << 51, (1 << 51) - 1], dtype=np.uint64)
    frac[: 200 * len(edge)] = np.tile(edge, 200)
    exp = rng.integers(1023 - 100, 1023 + 100, n).astype(np.uint64)
    exp[: 200 * len(edge)] = np.repeat(np.arange(1023 - 100, 1023 + 100, dtype=np.uint64), len(edge))
    b = ((exp << np.uint64(52)) | frac).view(np.float64)
    a = rng.standard_normal(n) * 10.0 ** rng.uniform(-20, 20, n)
    a[::97] = 0.0
    a[1::97] = b[1::97]
    y, q, ok, y0, q0 = kernels(a, b)
    ok = ok.astype(bool)
    assert np.array_equal(ok, (frac & np.uint64(0xffffffff)) != 0xffffffff)
    assert np.array_equal(y[ok], y0[ok])
    assert np.array_equal(q[ok], q0[ok])


def test_range(kernels):
    b = np.array([2.0 ** -100, 2.0 ** 100 * (1 - 2.0 ** -52), 2.0 ** -101, 2.0 ** 100, 0.0, -0.0, -1.0, np.inf, -np.inf,
                  np.nan, 5e-324])
    ok = kernels(np.ones_like(b), b)[2]
    assert ok.tolist() == [1, 1] + [0] * 9


def test_quotient_by_a_reciprocal_is_ieee_everywhere(kernels):
    """uw_quot with y = RN(1/b): the bits of a / b (signs of zeroes included) for numerators and divisors of
    any size, subnormal and infinite ones too."""
    rng = np.random.default_rng(3)
    n = 2_000_000
    a = rng.standard_normal(n) * 2.0 ** rng.uniform(-1070, 1020, n)
    b = rng.standard_normal(n) * 2.0 ** rng.uniform(-1070, 1020, n)
    near = rng.random(n) < 0.5
    a[near] = rng.standard_normal(near.sum()) * 2.0 ** rng.uniform(-420, 420, near.sum())
    b[near] = rng.standard_normal(near.sum()) * 2.0 ** rng.uniform(-30, 30, near.sum())
    special = np.array([0.0, -0.0, 1.0, -1.0, 5e-324, -5e-324, np.inf, -np.inf, np.nan, 2.0 ** -1022, 1.7e308, 2.0 - 2.0 ** -52])
    a[: len(special) ** 2] = np.repeat(special, len(special))
    b[: len(special) ** 2] = np.tile(special, len(special))
    q, q0 = kernels.quot(a, b)
    nan = np.isnan(q0)
    assert np.array_equal(np.isnan(q), nan)
    assert np.array_equal(q[~nan].view(np.int64), q0[~nan].view(np.int64))
