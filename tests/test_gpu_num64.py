"""The FP64 helpers of the sweeps on the device, over random operands of every
exponent that their domain holds and special values: the divisions by a
reciprocal (quotient(x, y, reciprocal(y))) against IEEE division, the integer
comparisons and tests against the plain ones, the truncation to FP32.

With e the relative error of the reciprocal, the corrected quotient is the
rounding of x / y (1 + d), |d| <= |e| (|e| + 2^-53) plus the remainder's rounding,
below 2^-102: the correctly rounded quotient unless x / y lies that close to the
middle of two numbers, which of random operands none in 2^48 does."""
import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "brx_num64.cuh"
using namespace brx;
__global__ void sweep(int n, const double *x, const double *y, double *r, double *q, float *t, int *flags)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        r[i] = reciprocal(y[i]);
        q[i] = quotient(x[i], y[i], r[i]);
        t[i] = truncated(x[i]);
        flags[i] = greater(x[i], y[i]) | negative(x[i]) << 1 | finite_bits(x[i]) << 2 |
                   (__double_as_longlong(unordered(ordered(x[i]))) == __double_as_longlong(x[i])) << 3;
    }
}
extern "C" int run(int n, const double *x, const double *y, double *r, double *q, float *t, int *flags)
{
    sweep<<<152, 256>>>(n, x, y, r, q, t, flags);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import torch

    from braids_hkt_gb300.build import ARCH, COMMON, CSRC, UNITS, nvcc
    folder = tmp_path_factory.mktemp("num64")
    source, library = folder / "num64.cu", folder / "num64.so"
    source.write_text(SOURCE)
    flags = dict(UNITS)["brx_api.cu"]
    subprocess.run([nvcc(), *ARCH, *COMMON, *flags, "-shared", f"-I{CSRC}", str(source), "-o", str(library)], check=True)
    lib = C.CDLL(str(library))

    def call(x, y):
        n = len(x)
        dx, dy = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y))
        r, q = torch.empty_like(dx), torch.empty_like(dx)
        t = torch.empty(n, dtype=torch.float32, device="cuda")
        flags = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lib.run(n, *(C.c_void_p(v.data_ptr()) for v in (dx, dy, r, q, t, flags))) == 0
        return tuple(v.cpu().numpy() for v in (r, q, t, flags))
    return call


def operands(rng, n, low, high, edge=False):
    """Random numbers of both signs with exponents low .. high - 1; edge: mantissas
    of up to four units in the last place from a power of two."""
    near = 1.0 + rng.integers(0, 5, n) * 2.0 ** -52, 2.0 - rng.integers(1, 5, n) * 2.0 ** -52
    mantissa = np.where(rng.random(n) < 0.5, *near) if edge else rng.uniform(1.0, 2.0, n)
    return rng.choice((-1.0, 1.0), n) * np.ldexp(mantissa, rng.integers(low, high, n))


@pytest.mark.parametrize("edge", [False, True])
def test_reciprocal_and_quotient(run, edge):
    rng = np.random.default_rng(3)
    n = 1 << 21
    y = operands(rng, n, -1020, 1021, edge)
    r, zero, _, _ = run(np.zeros(n), y)
    assert np.all(np.abs(r * y - 1.0) <= 2.0 ** -52)
    assert np.all(zero == 0.0)
    x, y = operands(rng, n, -450, 450, edge), operands(rng, n, -450, 450, edge)
    q = run(x, y)[1]
    if edge:                                    # quotients within 2^-104 of a middle are among these
        assert np.all(np.abs(q - x / y) <= np.spacing(np.abs(x / y)))
    else:
        np.testing.assert_array_equal(q, x / y)


def test_comparisons_and_truncation(run):
    rng = np.random.default_rng(9)
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 2.2e-308, -2.2e-308, 1.0, -1.0, 1.7976931348623157e308,
                        -1.7976931348623157e308, np.inf, -np.inf])
    a, b = np.meshgrid(special, special)
    x = np.concatenate((a.ravel(), operands(rng, 1 << 18, -1022, 1023)))
    y = np.concatenate((b.ravel(), operands(rng, 1 << 18, -1022, 1023)))
    _, _, t, flags = run(x, y)
    signed_zeros = (x == 0.0) & (y == 0.0)
    want = np.where(signed_zeros, np.signbit(y) & ~np.signbit(x), x > y)        # 0 above -0
    np.testing.assert_array_equal(flags & 1, want)
    np.testing.assert_array_equal(flags >> 1 & 1, x < 0.0)
    np.testing.assert_array_equal(flags >> 2 & 1, np.isfinite(x))
    assert np.all(flags >> 3 & 1)
    inside = (np.abs(x) >= 2.0 ** -126) & (np.abs(x) < 2.0 ** 128)
    err = np.abs(t[inside].astype(float) - x[inside])
    assert np.all(err < 2.0 ** -23 * np.abs(x[inside])) and np.all(np.abs(t[inside]) <= np.abs(x[inside]))
    assert np.all(t[np.abs(x) < 2.0 ** -126] == 0.0)
    nans = np.array([0x7ff8000000000000, 0xfff8000000000000, 0x7ff0000000000001, 0xffffffffffffffff], dtype=np.uint64)
    _, _, _, flags = run(nans.view(np.float64), np.zeros(4))
    assert np.all(flags >> 1 & 3 == 0)                                          # neither negative nor finite
