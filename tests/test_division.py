"""The branch-free division of the split search (csrc/division.cuh) against the operator, whose quotients are correctly
rounded: on the CPU (with another approximation to start from) and on the device."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-boost_b200", "csrc")

HOST = r"""
#include "division.cuh"
extern "C" int run(const double* a, const double* b, long long n, double* plain, double* op, unsigned char* ok) {
  for (long long i = 0; i < n; ++i) {
    ok[i]    = lbk::DivisionIsPlain(a[i], b[i]);
    plain[i] = lbk::DividePlain(a[i], b[i]);
    op[i]    = a[i] / b[i];
  }
  return 0;
}
"""
DEVICE = r"""
#include "division.cuh"
__global__ void k(const double* a, const double* b, long long n, double* plain, double* op, unsigned char* ok) {
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= n) return;
  ok[i]    = lbk::DivisionIsPlain(a[i], b[i]);
  plain[i] = lbk::DividePlain(a[i], b[i]);
  op[i]    = a[i] / b[i];
}
extern "C" int run(const double* a, const double* b, long long n, double* plain, double* op, unsigned char* ok) {
  double* d[4];
  unsigned char* f;
  for (int i = 0; i < 4; ++i)
    if (cudaMalloc(&d[i], 8 * n) != cudaSuccess) return 1;
  if (cudaMalloc(&f, n) != cudaSuccess) return 1;
  cudaMemcpy(d[0], a, 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d[1], b, 8 * n, cudaMemcpyHostToDevice);
  k<<<(unsigned)((n + 255) / 256), 256>>>(d[0], d[1], n, d[2], d[3], f);
  cudaMemcpy(plain, d[2], 8 * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(op, d[3], 8 * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(ok, f, n, cudaMemcpyDeviceToHost);
  for (int i = 0; i < 4; ++i) cudaFree(d[i]);
  cudaFree(f);
  return cudaGetLastError() != cudaSuccess;
}
"""


def operands(n):
    """Mantissas anywhere and within a few units of both ends, exponents anywhere and at both ends of the range, zeros,
    and operands that have to be refused."""
    rs = np.random.RandomState(7)

    def draw():
        m = rs.randint(0, 2 ** 52, size=n, dtype=np.int64)
        near = rs.randint(0, 8, size=n, dtype=np.int64)
        kind = rs.randint(0, 4, size=n)
        m = np.where(kind == 0, near, np.where(kind == 1, 2 ** 52 - 1 - near, m))
        e = np.where(rs.rand(n) < 0.5, rs.randint(523, 1523, size=n), rs.choice([523, 524, 1022, 1023, 1521, 1522], size=n))
        return ((e.astype(np.int64) << 52) | m).view(np.float64)

    a, b = draw(), draw()
    a[rs.rand(n) < 0.02] = 0.0
    odd = np.array([0.0, -1.0, np.inf, np.nan, 5e-324, 2.0 ** 500, 2.0 ** -501, np.nextafter(2.0 ** -500, 0), -(2.0 ** -300)])
    where = rs.rand(n) < 0.02
    b[where] = rs.choice(odd, size=int(where.sum()))
    where = rs.rand(n) < 0.02
    a[where] = rs.choice(odd[1:], size=int(where.sum()))
    # the quotients that a divisor of ones gives one unit off
    a[:1000] = 2.0 ** rs.randint(-499, 499, size=1000)
    b[:1000] = 2.0 ** rs.randint(-499, 499, size=1000) * (2.0 - 2.0 ** -52)
    return a, b


def check(run, n):
    a, b = operands(n)
    plain, op, ok = np.empty(n), np.empty(n), np.empty(n, dtype=np.uint8)
    rc = run(*(ctypes.c_void_p(t.ctypes.data) if not isinstance(t, int) else ctypes.c_longlong(t) for t in (a, b, n, plain, op, ok)))
    assert rc == 0
    ok = ok.astype(bool)
    in_range = (b >= 2.0 ** -500) & (b < 2.0 ** 500) & ((a == 0) | ((a >= 2.0 ** -500) & (a < 2.0 ** 500)))
    ones = (b.view(np.int64) & (2 ** 52 - 1)) == 2 ** 52 - 1
    assert np.array_equal(ok, in_range & ~ones)
    wrong = ok & (plain.view(np.int64) != op.view(np.int64))
    assert not wrong.any(), (a[wrong][:3], b[wrong][:3])
    with np.errstate(all="ignore"):
        assert np.array_equal(op[ok].view(np.int64), (a[ok] / b[ok]).view(np.int64))


def test_plain_division_rounds_correctly_on_the_cpu(tmp_path):
    (tmp_path / "d.cpp").write_text('#include <cmath>\n' + HOST)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-I", CSRC,
                    str(tmp_path / "d.cpp"), "-o", str(tmp_path / "d.so")], check=True)
    check(ctypes.CDLL(str(tmp_path / "d.so")).run, 2_000_000)


@pytest.mark.gpu
def test_plain_division_equals_the_operator_on_the_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    (tmp_path / "d.cu").write_text(DEVICE)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                    "-I", CSRC, str(tmp_path / "d.cu"), "-o", str(tmp_path / "d.so")], check=True)
    check(ctypes.CDLL(str(tmp_path / "d.so")).run, 20_000_000)
