"""The kernels' own quotients, reciprocals and square roots (common.cuh,
jacobi.cuh) against IEEE arithmetic: equal in the MLS rotations, whose values
agree with the CPU restatement bit for bit, also for the operands closest to a
rounding boundary; within one unit in the last place elsewhere."""
import ctypes
import random
import subprocess

import numpy as np
import pytest

from pacman_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "jacobi.cuh"
using namespace pacman_b200;
// The sine of the rotation that annihilates p in [[0, p], [p, h]]: p / h for the
// h beside which 100 p is lost to rounding.
__device__ double sine(double p, double h) {
  __shared__ double us[2][128], vs[2][128];
  const MlsColumn u{&us[0][threadIdx.x]}, v{&vs[0][threadIdx.x]};
  double a[3] = {0.0, p, h};
  u[0] = v[0] = v[1] = 0.0;
  u[1] = -1.0;
  mls_rotate<2, 0, 1>(a, u, v);
  return u[0];
}
__device__ double apply(int op, double a, double b) {
  double r = 0.0;
  switch (op) {
  case 0: r = recip(a); break;
  case 1: r = quot(a, b, recip(b)); break;
  case 2: r = root(a); break;
  case 3: r = root_mid(a); break;
  default: r = sine(a, b); break;
  }
  return r;
}
__global__ void k(int op, long n, const double *a, const double *b, double *o) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x)
    o[i] = apply(op, a[i], b[i]);
}
extern "C" int run(int op, long n, const double *a, const double *b, double *o) {
  double *d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * 3 * n) != cudaSuccess) return 1;
  cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k<<<1184, 128>>>(op, n, d, d + n, d + 2 * n);
  const cudaError_t e = cudaMemcpy(o, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return int(e);
}
"""
RECIP, QUOT, ROOT, ROOT_MID, SINE = range(5)
ONE = 1023 << 52


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("arithmetic")
    src, lib = d / "arithmetic.cu", d / "libarithmetic.so"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH, *build.FILE_FLAGS["mls.cu"], "-O3", "-std=c++17",
                    f"-I{build.CSRC}", "-shared", "-Xcompiler", "-fPIC", "-o", str(lib), str(src)],
                   check=True, capture_output=True)
    fn = ctypes.CDLL(str(lib)).run
    ptr = ctypes.POINTER(ctypes.c_double)

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
        out = np.empty_like(a)
        assert fn(op, ctypes.c_long(a.size), a.ctypes.data_as(ptr), b.ctypes.data_as(ptr),
                  out.ctypes.data_as(ptr)) == 0
        return out
    return call


def _bits(u):
    return np.asarray(u, dtype=np.uint64).view(np.float64)


def _random(rng, count, e0, e1):
    """Uniform mantissas, exponents in [e0, e1)."""
    e = rng.integers(e0 + 1023, e1 + 1023, count, dtype=np.uint64) << np.uint64(52)
    return _bits(e | rng.integers(0, 1 << 52, count, dtype=np.uint64))


def _near_all_ones(count):
    return _bits(np.uint64(ONE + (1 << 52) - 1) - np.arange(count, dtype=np.uint64))


def _ulps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64)).max()


def _hard_quotients(count):
    # 2^54 a = +-1 modulo b: a / b is as near to a midpoint as a quotient can be.
    rnd = random.Random(1)
    a, b = [1.0, 1.5], [2.0 - 2.0 ** -52] * 2
    while len(a) < count:
        if rnd.random() < 0.5:
            d = rnd.randrange(1 << 52, 1 << 53) | 1
        else:
            d = (1 << 53) - 1 - 2 * rnd.randrange(1 << rnd.randrange(1, 50))
        inv = pow(pow(2, 54, d), -1, d)
        for n in (inv, d - inv):
            if 2 * n >= d:
                a.append(float(n))
                b.append(float(d))
    return np.array(a), np.array(b)


def test_quotients_of_the_rotations(run):
    rng = np.random.default_rng(2)
    for a, b in (_hard_quotients(200_000),
                 (_random(rng, 1 << 21, 0, 1), _random(rng, 1 << 21, 0, 1)),
                 (np.ones(1 << 16), _near_all_ones(1 << 16))):
        a = a * 2.0 ** -70
        assert np.array_equal(run(SINE, a, b), a / b)


def _square_roots_modulo(c, n):
    """The odd s < 2^n with s^2 = c modulo 2^n, for c = 1 modulo 8."""
    s = 1
    for k in range(3, n):
        if (s * s - c) >> k & 1:
            s += 1 << (k - 1)
    m = 1 << n
    return {t % m for t in (s, -s, s + m // 2, -s + m // 2)}


def _hard_roots():
    # Every x in [1, 4) with x 2^104 = M^2 + M + j, M of 53 bits and |j| <= 16.
    xs = set()
    for j in range(-16, 17):
        c = 1 - 4 * j
        if c % 8 != 1:
            continue  # no odd square
        for n in (54, 55):  # x in [1, 2) has a spacing of 2^52, in [2, 4) of 2^53
            for s in _square_roots_modulo(c % (1 << n), n):
                M = (s - 1) // 2
                X = M * M + M + j
                if 1 << 52 <= M < 1 << 53 and 1 << 104 <= X < 1 << 106 and int(float(X)) == X:
                    xs.add(float(X) / 2.0 ** 104)
    assert {1.0 + 2.0 ** -52, 4.0 * (1.0 - 2.0 ** -53)} <= xs
    return np.array(sorted(xs))


def test_roots_are_correctly_rounded(run):
    rng = np.random.default_rng(3)
    k = np.arange(1 << 20)
    scale = np.ldexp(1.0, 2 * rng.integers(0, 66, 1 << 20))
    for x in (_hard_roots(), 1.0 + k * 2.0 ** -52, 4.0 - (k + 1) * 2.0 ** -51,
              1.0 + rng.random(1 << 20) ** 8, _random(rng, 1 << 21, 0, 132),
              rng.choice(_hard_roots(), 1 << 20) * scale):
        assert np.array_equal(run(ROOT_MID, x), np.sqrt(x))


def test_others_are_within_one_ulp(run):
    rng = np.random.default_rng(4)
    for d in (_random(rng, 1 << 21, -1000, 1000), _near_all_ones(1 << 16)):
        assert _ulps(run(RECIP, d), 1.0 / d) <= 1
        a = d[rng.permutation(d.size)] if d.max() < 2.0 else _random(rng, d.size, -20, 20)
        a = a * np.ldexp(1.0, np.clip(np.frexp(d)[1], -900, 900))
        assert _ulps(run(QUOT, a, d), a / d) <= 1
        assert np.array_equal(run(QUOT, d, d), np.ones_like(d))
    # Every normal number; the residual of the smallest is subnormal.
    x = np.r_[_random(rng, 1 << 21, -960, 1024), np.finfo(float).max]
    assert _ulps(run(ROOT, x), np.sqrt(x)) <= 1
    x = np.r_[_random(rng, 1 << 21, -1022, -960), np.finfo(float).tiny]
    assert _ulps(run(ROOT, x), np.sqrt(x)) <= 2
    x = np.array([0.0, 5e-324, np.nextafter(np.finfo(float).tiny, 0.0), np.inf, np.nan])
    assert np.array_equal(run(ROOT, x), np.array([0.0, 0.0, 0.0, np.inf, np.nan]), equal_nan=True)
