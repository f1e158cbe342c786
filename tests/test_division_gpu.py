"""The branch-free division of the per-point formulas, the stop rule without a
square root and the index division against what they stand for: `/`, sqrt and
integer division, bit for bit.  The device functions are compiled from the
library's own sources with its own flags.

Divisors: random, powers of two, and significands up to 3000 units below all
ones (Markstein's exception and its neighbours, where a reciprocal that is not
rounded to nearest gives a wrong quotient), each with the numerators whose
quotients lie next to a rounding boundary, and both ends of the exponent
range.  Divisors are positive, as all of the solvers' are (div_uniform takes
any)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from coldplate_solver_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "cps_thermal.cu"
__global__ void divide(long long n, const double* a, const double* b, const double* u, double* out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    out[k] = cps::div_rn(a[k], b[k]);
    out[n + k] = cps::recip(b[k]);
    out[2 * n + k] = cps::div_uniform(a[k], b[k]);
    const double c = b[k] / u[k];  // a relaxed diagonal: its reciprocal from the diagonal's
    out[3 * n + k] = cps::div_rn(a[k], c, cps::recip_from(c, u[k] * cps::recip(b[k])));
    out[4 * n + k] = a[k] / c;
  }
}
// per significand that the approximation tells apart (the upper 20 bits): the largest relative error at exponent
// 2^e, with the lower word all zeros or all ones, and whether the uppermost one's is the power of two
__global__ void approximation(int e, double* err, int* power) {
  const int hi = ((1023 + e) << 20) | (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const double b0 = __hiloint2double(hi, 0), b1 = __hiloint2double(hi, -1);
  const double y0 = cps::recip_approx(b0), y1 = cps::recip_approx(b1);
  err[hi & 0xfffff] = y0 == y1 ? fmax(fabs(__fma_rn(-b0, y0, 1.0)), fabs(__fma_rn(-b1, y1, 1.0))) : 1.0;
  if ((hi & 0xfffff) == 0xfffff) *power = y1 == ldexp(1.0, -e - 1);
}
__global__ void index_divide(cpt::FastDiv f, int n, const int* x, int* out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) out[k] = f(x[k]);
}
extern "C" int run_divide(long long n, const double* a, const double* b, const double* u, double* out) {
  divide<<<296, 256>>>(n, a, b, u, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_approximation(int e, double* err, int* power) {
  approximation<<<4096, 256>>>(e, err, power);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_index_divide(int d, int n, const int* x, int* out) {
  index_divide<<<148, 256>>>(cpt::FastDiv::of(d), n, x, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" double stop_of(double tol) { return cps::pcg_stop(tol); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("division")
    src, so = tmp / "division.cu", tmp / "division.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", os.path.join(build.PKG_DIR, "csrc"), "-o", str(so), str(src)],
                   check=True)
    h = ctypes.CDLL(str(so))
    p = ctypes.c_void_p
    h.run_divide.argtypes = [ctypes.c_longlong, p, p, p, p]
    h.run_approximation.argtypes = [ctypes.c_int, p, p]
    h.run_index_divide.argtypes = [ctypes.c_int, ctypes.c_int, p, p]
    h.stop_of.argtypes, h.stop_of.restype = [ctypes.c_double], ctypes.c_double
    return h


def same_bits(x, y):
    nan = np.isnan(x) & np.isnan(y)
    bad = np.flatnonzero(~nan & (x.view(np.uint64) != y.view(np.uint64)))
    return bad


def check(lib, a, b, only=("div_rn", "recip", "div_uniform", "relaxed")):
    import torch
    a, b = np.broadcast_arrays(np.asarray(a, np.float64), np.asarray(b, np.float64))
    a, b = np.ascontiguousarray(a).ravel(), np.ascontiguousarray(b).ravel()
    n = len(a)
    u = np.random.default_rng(n).uniform(0.05, 1.0, n)
    dev = [torch.from_numpy(x).cuda() for x in (a, b, u)]
    out = torch.empty(5 * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_divide(n, *[x.data_ptr() for x in dev], out.data_ptr()) == 0
    out = out.cpu().numpy().reshape(5, n)
    with np.errstate(all="ignore"):
        want = {"div_rn": (out[0], a / b), "recip": (out[1], 1.0 / b), "div_uniform": (out[2], a / b),
                "relaxed": (out[3], out[4])}
    for name in only:
        bad = same_bits(*want[name])
        assert len(bad) == 0, (name, len(bad), [(float.hex(a[k]), float.hex(b[k])) for k in bad[:4]])


def boundary_pairs(divisors, rng):
    """a, b with a / b within a few units of 2^-53 of the middle of two neighbouring values: for an odd
    53-bit b, A 2^e = b m + s with an odd 54-bit m and a small odd s."""
    a, b = [], []
    for d in divisors:
        for e in (53, 54):
            for s in (-3, -1, 1, 3):
                m = (-s * pow(d, -1, 1 << e)) % (1 << e)
                num = d * m + s
                if m & 1 and num % (1 << e) == 0 and 0 < num >> e < 1 << 53:
                    a.append(num >> e)
                    b.append(d)
    return np.array(a, np.float64), np.array(b, np.float64)


@pytest.mark.parametrize("e", [-1000, -34, -1, 0, 1, 52, 999])
def test_reciprocal_approximation(lib, e):
    import torch
    err = torch.empty(1 << 20, dtype=torch.float64, device="cuda")
    power = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_approximation(e, err.data_ptr(), power.data_ptr()) == 0
    assert err.max().item() < 2.0 ** -18.5
    assert power.item() == 1


def test_division_random(lib):
    rng = np.random.default_rng(1)
    n = 4_000_000
    scale = lambda lo, hi: np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n))  # noqa: E731
    check(lib, scale(-20, 20) * rng.choice([-1.0, 1.0], n), scale(-30, 30))
    check(lib, scale(-20, 20), -scale(-30, 30), only=("div_uniform",))
    check(lib, scale(-300, 300), scale(-300, 300))


def test_division_next_to_rounding_boundaries(lib):
    rng = np.random.default_rng(2)
    near = [(1 << 53) - k for k in range(1, 6001, 2)]
    other = [int(x) | 1 for x in rng.integers(1 << 52, 1 << 53, 20000)]
    a, b = boundary_pairs(near + other, rng)
    assert len(a) > 20000
    check(lib, a, b)
    check(lib, np.ldexp(a, -60), np.ldexp(b, -90))


def test_division_edges_of_the_significand(lib):
    k = np.arange(300)
    low, high = 2.0 ** 52 + k, 2.0 ** 53 - k
    x = np.concatenate([low, high])
    check(lib, x[:, None], x[None, :])
    check(lib, -x[:, None], np.ldexp(x, -70)[None, :])


def test_division_zeros_infinities_and_the_ends_of_the_range(lib):
    b = np.ldexp([1.0, 1.5, 2 - 2.0 ** -52, 4 / 3], [[-1000], [-500], [0], [500], [999]]).ravel()
    numerators = np.array([0.0, -0.0, np.inf, -np.inf, np.nan])[:, None]
    check(lib, numerators, b[None, :], only=("div_rn", "recip", "div_uniform"))
    check(lib, numerators, -b[None, :], only=("div_uniform",))
    a = np.ldexp(np.array([1.0, 1.9, 2 - 2.0 ** -52]), [[-960], [0], [1000]]).ravel()
    a, d = [x.ravel() for x in np.broadcast_arrays(np.concatenate([a, -a])[:, None], b[None, :])]
    with np.errstate(all="ignore"):
        keep = ~((np.abs(a / d) < 2.0 ** -1021))
    check(lib, a[keep], d[keep], only=("div_rn", "div_uniform"))
    # every operand: div_uniform
    special = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0 ** -1022, 1.7e308, np.inf, np.nan, 3.0])
    check(lib, special[:, None], special[None, :], only=("div_uniform",))


def test_pcg_stop_is_the_square_root_test(lib):
    rng = np.random.default_rng(3)
    for tol in [1e-6, 1e-5, 1e3, 1.0, 2 - 2.0 ** -52, 1e-160, 1e-200, 1e200, *10.0 ** rng.uniform(-12, 3, 200)]:
        x = lib.stop_of(tol)
        assert np.sqrt(x) >= tol and (x == 0.0 or np.sqrt(np.nextafter(x, 0.0)) < tol), tol
    for tol in (0.0, -1.0, float("nan")):
        assert lib.stop_of(tol) == 0.0


def test_index_division_is_exact(lib):
    import torch
    rng = np.random.default_rng(4)
    top = (1 << 31) - 1
    for d in [1, 2, 3, 5, 7, 31, 32, 33, 125, 250, 1000, 4096, 31250, 65535, 65536, 500000, (1 << 30) - 1, 1 << 30]:
        q = np.concatenate([rng.integers(0, top // d + 1, 20000), np.arange(min(2000, top // d + 1)),
                            [top // d]]).astype(np.int64) * d
        x = np.unique(np.clip(np.concatenate([q - 1, q, q + 1, rng.integers(0, top, 20000), [top]]), 0, top))
        dev = torch.from_numpy(x.astype(np.int32)).cuda()
        out = torch.empty_like(dev)
        torch.cuda.synchronize()
        assert lib.run_index_divide(d, len(x), dev.data_ptr(), out.data_ptr()) == 0
        assert np.array_equal(out.cpu().numpy(), x // d), d
