"""The integer-pipe forms of FP64 operations (fp64_tools.cuh, the cells of
mpm_axis.cuh) against IEEE arithmetic: to the bit, or by value for a zero's sign
where the form gives up that; roots and their reciprocals within one unit in the
last place. Operands: zeros, subnormals, powers of two and their neighbours, the
ends of FP64's, FP32's and the integers' ranges, halves and rounding ties,
infinities, NaN, mantissas of all ones, and a million at random."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from libhybridgrains_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "hg_internal.cuh"
#include "mpm_axis.cuh"
using namespace hg;
__global__ void k(int op, int n, const double *a, const double *b, double *x, double *y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double u = a[i], w = b[i];
  double r = 0.0, s = 0.0;
  if (op == 0) r = twice(u);
  if (op == 1) r = halved(u);
  if (op == 2) r = min_zero(u);
  if (op == 3) r = (double)narrow(u);
  if (op == 4) r = widen_f32((float)u);
  if (op == 5) { r = (double)floor_int(u); s = (double)ceil_int(u); }
  if (op == 6) r = index_f64((int)u);
  if (op == 7) r = quot(u, divisor(w));
  if (op == 8) { const double2 q = root(u); r = q.x; s = q.y; }
  if (op == 9) {
    bool ok = true;
    const Divisor H = divisor(w);
    Cells c = cells<false>(u, H, ok);
    if (!ok || !H.ok) c = cells<true>(u, H, ok);
    r = (double)c.lo;
    s = (double)c.hi;
  }
  if (op == 10) { r = f64_zero(u); s = finite_bits(u); }
  if (op == 11) r = f64_less(fabs(u), fabs(w));
  if (op == 12) r = (double)narrow_trunc(u);
  x[i] = r;
  y[i] = s;
}
extern "C" int run(int op, int n, const double *a, const double *b, double *x, double *y) {
  double *d = nullptr;
  const size_t s = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 4 * s) != cudaSuccess) return 1;
  cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(op, n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
  cudaMemcpy(x, d + 2 * (size_t)n, s, cudaMemcpyDeviceToHost);
  cudaMemcpy(y, d + 3 * (size_t)n, s, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def tool(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64_tools")
    src, lib = str(d / "t.cu"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", build.INCLUDE, "-I", build.CSRC, src, "-o", lib],
                   check=True, capture_output=True)
    run = ctypes.CDLL(lib).run

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ascontiguousarray(a if b is None else b, dtype=np.float64)
        x, y = np.empty_like(a), np.empty_like(a)
        p = [v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, x, y)]
        assert run(op, len(a), *p) == 0
        return x, y
    return call


def edges():
    e = np.arange(-1074, 1024)
    p = np.ldexp(1.0, e)
    near = np.concatenate([p, np.nextafter(p, 0.0), np.nextafter(p, np.inf), 1.5 * p,
                           np.nextafter(1.5 * p, 0.0)])
    # FP32 rounding ties, and their neighbours
    m = np.ldexp(1.0 + (2.0 * np.arange(64) + 1.0) * 2.0 ** -24, np.arange(-160, 160)[:, None])
    m = m.ravel()
    near = np.concatenate([near, m, np.nextafter(m, 0.0), np.nextafter(m, np.inf),
                           np.arange(300) * 0.5, [0.0, np.finfo(float).max, np.inf]])
    rng = np.random.default_rng(1)
    r = np.ldexp(rng.uniform(1.0, 2.0, 500000), rng.integers(-1070, 1023, 500000))
    c = np.ldexp(rng.uniform(1.0, 2.0, 500000), rng.integers(-40, 40, 500000))
    a = np.concatenate([near, r, c])
    return np.concatenate([a, -a, [np.nan]])


def bits(x):
    return x.view(np.int64)


def test_conversions_and_scalings(tool):
    a = edges()
    with np.errstate(all="ignore"):
        for op, want in ((0, 2.0 * a), (1, 0.5 * a), (3, a.astype(np.float32).astype(float)),
                         (4, a.astype(np.float32).astype(float))):
            got = tool(op, a)[0]
            bad = (bits(got) != bits(want)) & ~(np.isnan(got) & np.isnan(want))
            assert not bad.any(), (op, a[bad][:5], got[bad][:5], want[bad][:5])
    assert np.array_equal(tool(2, a)[0], np.where(a < 0.0, a, 0.0))
    z, f = tool(10, a)
    assert np.array_equal(z, a == 0.0) and np.array_equal(f, np.isfinite(a))
    w = np.random.default_rng(2).permutation(a)
    ok = ~(np.isnan(a) | np.isnan(w))
    assert np.array_equal(tool(11, a, w)[0][ok], np.abs(a[ok]) < np.abs(w[ok]))
    # truncated where FP32 has a normal number: towards zero, by less than a unit
    t = a[(np.abs(a) >= 2.0 ** -126) & (np.abs(a) < 2.0 ** 127)]
    lo = t.astype(np.float32).astype(float)
    over = np.abs(lo) > np.abs(t)
    lo[over] = np.nextafter(lo[over].astype(np.float32), np.float32(0.0)).astype(float)
    assert np.array_equal(tool(12, t)[0], lo)


def test_integers(tool):
    a = edges()
    a = a[np.abs(a) < 2.0 ** 31 - 1]
    lo, hi = tool(5, a)
    assert np.array_equal(lo, np.floor(a)) and np.array_equal(hi, np.ceil(a))
    i = np.concatenate([np.arange(70000), 2 ** np.arange(31), 2 ** np.arange(1, 32) - 1,
                        np.random.default_rng(3).integers(0, 2 ** 31, 200000)]).astype(float)
    assert np.array_equal(bits(tool(6, i)[0]), bits(i))


def operands():
    """Quotients near and far from rounding boundaries."""
    rng = np.random.default_rng(4)
    k = np.arange(64)
    m = np.concatenate([1.0 + k * 2.0 ** -52, 2.0 - (k + 1) * 2.0 ** -52, 1.0 + 2.0 ** -(k % 52.0),
                        np.sqrt(1.0 + k / 64.0), 1.0 + rng.random(64)])
    a, b = np.meshgrid(m, m)
    a, b = a.ravel(), b.ravel()
    # a = q b rounded, from q half way between numbers: the hardest quotients
    q = rng.uniform(1.0, 2.0, 400000)
    d = rng.uniform(1.0, 2.0, 400000)
    h = q * d + np.spacing(q) * 0.5 * d
    a = np.concatenate([a, h, rng.uniform(1.0, 2.0, 400000), np.zeros(4)])
    b = np.concatenate([b, d, rng.uniform(1.0, 2.0, 400000), m[:4]])
    ea, eb = rng.integers(-30, 30, len(a)), rng.integers(-30, 30, len(a))
    far = rng.integers(0, 20, len(a)) == 0
    ea[far], eb[far] = rng.integers(-1060, 1020, far.sum()), rng.integers(-1060, 1020, far.sum())
    s = np.where(rng.integers(0, 2, len(a)) == 0, -1.0, 1.0)
    return np.ldexp(s * a, ea), np.ldexp(b, eb)


def test_quotients(tool):
    a, b = operands()
    with np.errstate(all="ignore"):
        want = a / b
    got = tool(7, a, b)[0]
    bad = got != want
    assert not bad.any(), (int(bad.sum()), a[bad][:5], b[bad][:5], got[bad][:5], want[bad][:5])


def test_roots(tool):
    a = np.abs(edges())
    a = np.concatenate([a[np.isfinite(a) & (a > 0.0)], operands()[1]])
    g, y = tool(8, a)
    with np.errstate(all="ignore"):
        s = np.sqrt(a)
        ext = np.sqrt(a.astype(np.longdouble))
    assert (np.abs(g - s) <= np.spacing(s)).all()
    inv = (1.0 / ext).astype(float)
    assert (np.abs(y - inv) <= 2.0 * np.spacing(inv)).all()
    assert (g != s).mean() < 1e-6


@pytest.mark.parametrize("h", [1.0e-3, 2.5e-3, 5.0e-3, 0.3, 1.0, 7.0])
def test_cells(tool, h):
    rng = np.random.default_rng(5)
    k = np.arange(-200, 5000)
    x = np.concatenate([k * h, np.nextafter(k * h, np.inf), np.nextafter(k * h, -np.inf),
                        k * h + 1.0e-9 * h, rng.uniform(-10.0, 2000.0, 300000) * h,
                        rng.uniform(0.0, 2.0 ** 22, 100000) * h])
    z = x / h
    lo, hi = tool(9, x, np.full(len(x), h))
    assert np.array_equal(lo, np.floor(z))
    whole = np.floor(z) == z
    assert np.array_equal(hi[~whole], np.ceil(z[~whole])) and np.array_equal(hi[whole], z[whole])
