"""The FP64 passes' own arithmetic, function by function: square root, quotient and reciprocal square root by
Newton's iteration, the singular kernels' power by table, and the integer sums. The functions are compiled from
their headers into a small library here and compared elementwise with extended precision."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "geometry.cuh"
#include "primitives.cuh"
#include "quadrature.cuh"
#include "passes.cuh"
#include "passes_mix.cuh"
#include "passes_f64.cuh"
using namespace nlg;
__global__ void k_math(int op, long n, const double *a, const double *b, const double *tab, double *o, long long *i3) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (op == 0) o[i] = f64_sqrt(a[i]);
    if (op == 1) o[i] = f64_div(a[i], b[i]);
    if (op == 2) o[i] = f64_rsqrt(a[i]);
    if (op == 3) o[i] = pw_eval(tab, a[i]);
    if (op == 4) {
        bool bad = false, rest = false;
        f64_split(a[i], F64_BITS, bad, i3[4 * i], i3[4 * i + 1], rest);
        i3[4 * i + 2] = rest ? f64_third(a[i]) : 0;
        i3[4 * i + 3] = bad;
    }
    if (op == 5) o[i] = f64_join(i3[4 * i], i3[4 * i + 1], i3[4 * i + 2]);
}
extern "C" int run(int op, long n, const double *a, const double *b, double kc, double expo, double *o, long long *i3) {
    double *d[4] = {nullptr, nullptr, nullptr, nullptr};
    long long *di = nullptr;
    ProbParams P, *dp = nullptr;
    memset(&P, 0, sizeof(P));
    P.kc = kc; P.expo = expo; P.singular = 1;
    const size_t by[4] = {n * 8ul, n * 8ul, n * 8ul, PW_N * 8ul};
    bool ok = cudaMalloc(&dp, sizeof(P)) == cudaSuccess && cudaMalloc(&di, n * 32) == cudaSuccess;
    for (int k = 0; k < 4; k++) ok = ok && cudaMalloc(&d[k], by[k]) == cudaSuccess;
    if (ok) {
        cudaMemcpy(d[0], a, n * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(d[1], b, n * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(di, i3, n * 32, cudaMemcpyHostToDevice);
        cudaMemcpy(dp, &P, sizeof(P), cudaMemcpyHostToDevice);
        k_pw_table<<<(PW_N + 63) / 64, 64>>>(dp, 1, d[3]);
        k_math<<<(unsigned)((n + 127) / 128), 128>>>(op, n, d[0], d[1], d[3], d[2], di);
        cudaMemcpy(o, d[2], n * 8, cudaMemcpyDeviceToHost);
        cudaMemcpy(i3, di, n * 32, cudaMemcpyDeviceToHost);
    }
    ok = ok && cudaDeviceSynchronize() == cudaSuccess;
    for (double *p : d) cudaFree(p);
    cudaFree(di);
    cudaFree(dp);
    return ok ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from nlfem_gb300 import build
    d = tmp_path_factory.mktemp("f64math")
    (d / "m.cu").write_text("#include <cstring>\n" + SOURCE)
    subprocess.run([build.NVCC] + build.ARCH + ["-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", build.CSRC,
                    "-I", os.path.join(ROOT, "include"), "-o", str(d / "m.so"), str(d / "m.cu")], check=True)
    lib = ctypes.CDLL(str(d / "m.so"))
    dp = ctypes.POINTER(ctypes.c_double)
    lib.run.argtypes = [ctypes.c_int, ctypes.c_long, dp, dp, ctypes.c_double, ctypes.c_double, dp, ctypes.POINTER(ctypes.c_longlong)]

    def call(op, a, b=None, kc=1.0, expo=0.0, i3=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.zeros_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
        i3 = np.zeros((len(a), 4), dtype=np.int64) if i3 is None else np.ascontiguousarray(i3)
        o = np.zeros_like(a)
        assert lib.run(op, len(a), a.ctypes.data_as(dp), b.ctypes.data_as(dp), kc, expo, o.ctypes.data_as(dp),
                       i3.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))) == 0
        return o, i3
    return call


def _samples(lo, hi, per, seed):
    """Random mantissas in every binade of [2^lo, 2^hi), the powers of two and their neighbours."""
    rng = np.random.Generator(np.random.PCG64(seed))
    e = np.repeat(np.arange(lo, hi), per)
    v = np.ldexp(1.0 + rng.random(len(e)), e)
    p = np.ldexp(1.0, np.arange(lo + 1, hi))
    return np.concatenate([v, p, np.nextafter(p, 0), np.nextafter(p, np.inf)])


def _ulps(got, want):
    """Error in units of the last place of want (extended precision)."""
    w = want.astype(np.float64)
    return np.abs((got.astype(np.longdouble) - want) / np.spacing(np.abs(w))).astype(float)


# The last Newton step is a residual correction whose own rounding is half a unit: one unit bounds the square root
# and the quotient; the reciprocal square root's last step has three roundings (two units). All exponents: the
# seeds serve 2^-98 to 2^98, CUDA's routines the rest.
def test_sqrt(run):
    a = _samples(-1000, 1000, 40, 1)
    assert _ulps(run(0, a)[0], np.sqrt(a.astype(np.longdouble))).max() <= 1.0


def test_reciprocal_sqrt(run):
    a = _samples(-1000, 1000, 40, 2)
    assert _ulps(run(2, a)[0], 1 / np.sqrt(a.astype(np.longdouble))).max() <= 2.0


def test_quotient(run):
    b = _samples(-600, 600, 60, 3)
    rng = np.random.Generator(np.random.PCG64(4))
    a = np.ldexp(rng.choice([-1.0, 1.0], len(b)) * (1 + rng.random(len(b))), rng.integers(-200, 200, len(b)))
    b *= rng.choice([-1.0, 1.0], len(b))
    assert _ulps(run(1, a, b)[0], a.astype(np.longdouble) / b).max() <= 1.0


# Table entries of one unit each, the argument's reduced part, the series and the last product: 3 units or
# 6.7e-16. Arguments in every binade, and at and beside each of the table's 512 intervals' ends.
@pytest.mark.parametrize("expo", [1.0, 2.2, 2.8, 3.0, 3.8])
def test_power_table(run, expo):
    m = 1.0 + np.arange(512) / 512
    edges = np.concatenate([np.ldexp(x, k) for k in (-43, -20, -1, 0) for x in (m, np.nextafter(m, 0), np.nextafter(m, 2))])
    r2 = np.concatenate([_samples(-300, 20, 200, 5), edges])
    got = run(3, r2, kc=0.7, expo=expo)[0]
    want = np.longdouble(0.7) * r2.astype(np.longdouble) ** (np.longdouble(-0.5) * np.longdouble(expo))
    assert float(np.abs(got.astype(np.longdouble) / want - 1).max()) < 6.7e-16
    assert np.all(np.isinf(run(3, [0.0, 5e-324], kc=0.7, expo=expo)[0]))


# The parts of a number add up to it, exactly down to 2^-80, are of its sign, and their sums come back as one number.
def test_integer_parts(run):
    rng = np.random.Generator(np.random.PCG64(6))
    a = _samples(-140, 62, 30, 7)
    a = np.concatenate([a[a < 2.0 ** 62] * rng.choice([-1.0, 1.0], np.count_nonzero(a < 2.0 ** 62)), [0.0, 1.5, -0.75]])
    parts = run(4, a)[1]
    assert not parts[:, 3].any()
    for x, (hi, lo, third, _) in zip(a, parts.tolist()):
        s = Fraction(hi) + Fraction(lo, 1 << 40) + Fraction(third, 1 << 80)
        assert hi * x >= 0 and lo * x >= 0 and third * x >= 0
        assert (s != 0) == (x != 0)
        assert s == Fraction(x) or abs(s - Fraction(x)) < Fraction(1, 1 << 80)
    assert run(4, [2.0 ** 62, -(2.0 ** 62), np.inf, np.nan])[1][:, 3].all()
    # sums of parts of both signs
    i = rng.integers(0, len(a), (2000, 5))
    tot = np.array([[sum(int(parts[k, q]) for k in row) for q in range(3)] + [0] for row in i])
    keep = np.abs(tot[:, 0]) < 2 ** 62
    got = run(5, np.zeros(keep.sum()), i3=tot[keep].astype(np.int64))[0]
    for g, (hi, lo, third, _) in zip(got, tot[keep].tolist()):
        s = Fraction(hi) + Fraction(lo, 1 << 40) + Fraction(third, 1 << 80)
        # two roundings of the larger parts; what cancels between the parts cancels exactly
        assert abs(Fraction(g) - s) <= abs(s) * Fraction(3, 1 << 53)
