"""The reciprocal of the FP64 saturation adjustment (uw_rcp, compiled from the kernel's header by itself)
and the division built on it (uw_div_by) against the GPU's IEEE division: every bit, over the whole range
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
    column = open(os.path.join(CSRC, "uwshcu_fp64_kernel.cuh")).read()
    math = open(os.path.join(CSRC, "uw_math.h")).read()
    src = ("#define UW_MUL(a, b) __dmul_rn((a), (b))\n" + _function(column, "__device__ __forceinline__ double uw_rcp(")
           + _function(column, "__device__ __forceinline__ bool uw_rcp_ok(") + "\n__device__ " + _function(math, "UW_HD double uw_div_by(")
           + """
extern "C" __global__ void rcp_kernel(const double* a, const double* b, double* y, double* q, int* ok, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = uw_rcp(b[i]);
    q[i] = uw_div_by(a[i], b[i], y[i]);
    ok[i] = uw_rcp_ok(b[i]);
}
""")
    k = torch.cuda._compile_kernel(src, "rcp_kernel")

    def run(a, b):
        a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        y, q = torch.empty_like(b), torch.empty_like(b)
        ok = torch.empty(b.shape, dtype=torch.int32, device="cuda")
        n = b.numel()
        k(grid=((n + 255) // 256, 1, 1), block=(256, 1, 1), args=(a, b, y, q, ok, n))
        return [t.cpu().numpy() for t in (y, q, ok, 1.0 / b, a / b)]
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
