"""The FP64 bond loop's root and quotient (pdgpu_quot.cuh) against sqrt and
division, with the reciprocals the loop hands them: on random operands, and on
operands whose exact result lies next to the midpoint of two doubles.

With b, m integers of 53 and 54 bits, m odd, and a 2^54 = b m + t, the quotient
a / b is off a midpoint by the relative t / (b m); with a 2^55 = m m + t the
root of a by t / (2 m m).  The last correction is off by at most 12 2^-106 of the
result (quotient: 3 2^-53 in the reciprocal times 4 2^-53 in the first
quotient; root: less), so from |t| = 32 on (root: 64) the result is the rounded
one, and below that its neighbour at most.  With 1 / b itself rounded it is the
rounded one throughout (Markstein).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "pdgpu_quot.cuh"
// out: root of b; 1 / sqrt(b) as the loop has it; a / sqrt(b); a / b by the squared reciprocal and by 1 / b
__global__ void k(const double *a, const double *b, double *out, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const pdgpu::Root R = pdgpu::root(b[i]);
  out[i] = R.r;
  out[n + i] = pdgpu::quot(a[i], R.r, R.inv);
  out[2 * n + i] = pdgpu::quot(a[i], b[i], R.inv * R.inv);
  out[3 * n + i] = pdgpu::quot(a[i], b[i], 1.0 / b[i]);
}
extern "C" int quot_check(const double *a, const double *b, double *out, int n) {
  double *d;
  if (cudaMalloc(&d, 6 * n * sizeof(double)) != cudaSuccess) return -1;
  cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
  cudaMemcpy(out, d + 2 * n, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from peridem_b200 import build
    d = tmp_path_factory.mktemp("quot")
    src, lib = str(d / "quot.cu"), str(d / "quot.so")
    with open(src, "w") as fh:
        fh.write(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "-I", build.CSRC, "-o", lib, src], check=True)
    f = ctypes.CDLL(lib).quot_check

    def call(a, b):
        a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b))
        out = np.empty((4, a.size))
        p = [v.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for v in (a, b, out)]
        assert f(*p, ctypes.c_int(a.size)) == 0
        return out
    return call


def _ulps(got, want):
    return np.abs(got.view(np.int64) - want.view(np.int64))


@pytest.mark.parametrize("span", [0, 40, 300])
def test_random_operands(check, span):
    rng = np.random.default_rng(span)
    n = 4_000_000
    b = np.ldexp(1.0 + rng.random(n), rng.integers(-span, span + 2, n).astype(np.int32))
    a = np.ldexp(1.0 + rng.random(n), rng.integers(-span, span + 2, n).astype(np.int32)) * rng.choice([-1.0, 1.0], n)
    r, ar, ab2, ab = check(a, b)
    assert np.array_equal(r, np.sqrt(b))
    assert np.array_equal(ar, a / np.sqrt(b))
    assert np.array_equal(ab2, a / b) and np.array_equal(ab, a / b)


def _next_to_midpoints(rng, offsets, count):
    """a, b with a 2^54 = b m + t, m odd of 54 bits, and t."""
    a, b, t = [], [], []
    for off in offsets:
        k = 0
        while k < count:
            bi = int(rng.integers(1 << 52, 1 << 53)) | 1
            ti = off if rng.random() < 0.5 else -off
            m = -ti * pow(bi, -1, 1 << 54) % (1 << 54)
            ai = (bi * m + ti) >> 54
            if m < 1 << 53 or not 1 << 52 <= ai < 1 << 53:
                continue
            assert ai << 54 == bi * m + ti and m % 2
            a.append(float(ai)), b.append(float(bi)), t.append(off)
            k += 1
    return np.array(a), np.array(b), np.array(t)


def test_quotients_next_to_midpoints(check):
    rng = np.random.default_rng(1)
    a, b, t = _next_to_midpoints(rng, (1, 3, 7, 15, 33, 65, 257, 4097), 4000)
    want = a / b
    _, _, ab2, ab = check(a, b)
    assert np.array_equal(ab, want)
    off = _ulps(ab2, want)
    print("neighbours of the rounded quotient:", {int(k): int(off[t == k].sum()) for k in np.unique(t)})
    assert off.max() <= 1 and not off[t >= 32].any()


def test_roots_next_to_midpoints(check):
    """m of 54 bits with m m = -t modulo 2^55, from the roots modulo 8 up."""
    b, t = [], []
    for ti in (s * k for k in range(1, 4096, 2) for s in (1, -1)):
        if -ti % 8 != 1:
            continue
        roots = [1, 3, 5, 7]
        for e in range(4, 56):
            roots = [r for q in roots for r in (q, q + (1 << (e - 1))) if (r * r + ti) % (1 << e) == 0]
            roots = sorted(set(roots))[:8]
        for m in roots:
            bi, rest = divmod(m * m + ti, 1 << 55)
            if 1 << 53 <= m < 1 << 54 and not rest and 1 << 52 <= bi < 1 << 53:
                b.append(float(bi)), t.append(abs(ti))
    b, t = np.array(b), np.array(t)
    assert b.size > 200 and t.min() < 16
    for even in (0, 2):  # the same mantissas at another even exponent
        x = np.ldexp(b, -40 - even)
        # b = m m 2^-55 needs an odd power of two: sqrt(2 b') with b' = b / 2
        got, want = check(np.ones_like(x), x * 2.0)[0], np.sqrt(x * 2.0)
        off = _ulps(got, want)
        print("neighbours of the rounded root:", int(off.sum()), "of", b.size)
        assert off.max() <= 1 and not off[t >= 64].any()
