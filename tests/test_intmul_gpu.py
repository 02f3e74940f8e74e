"""The trellis kernels' products on the integer pipe (csrc/sdm_intmul.h) against
the FP64 product, bit for bit: a small check kernel, compiled here from that
header, over operands built to meet every rounding (exact ties to even and odd,
a sticky bit in the lowest word alone, carries through the whole mantissa into
the exponent, both normalisations, the ends of the operands' range, signed
zeros) and over random ones."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SOURCE = r"""
#include "sdm_intmul.h"
using namespace dsdgpu;
__global__ void check(const IntCoef* c, const double* cv, int nc, const double* s, long long ns, int pairs,
                      unsigned long long* out) {
  const long long total = pairs ? ns : ns * nc;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long j = pairs ? i : i / nc;
    const int k = (int)(i % nc);
    const double x = s[j], want = __dmul_rn(cv[k], x);
    const long long w = __double_as_longlong(want);
    if (range_word(x) <= kRangeSpan) {
      atomicAdd(out + 0, 1ull);
      if (__double_as_longlong(int_mul(c[k], x)) != w) atomicAdd(out + 1, 1ull);
    }
    if (range_word0(x) <= kRangeSpan) {
      atomicAdd(out + 2, 1ull);
      if (__double_as_longlong(int_mul0(c[k], x)) != w) atomicAdd(out + 3, 1ull);
    }
  }
}
extern "C" int run(const double* c, int nc, const double* s, long long ns, int pairs, unsigned long long* out) {
  IntCoef* hc = new IntCoef[nc];
  for (int i = 0; i < nc; i++)
    if (!int_coef(c[i], hc + i)) return -1;
  IntCoef* dc; double *dv, *ds; unsigned long long* d;
  if (cudaMalloc(&dc, sizeof(IntCoef) * nc) || cudaMalloc(&dv, 8 * nc) || cudaMalloc(&ds, 8 * ns) || cudaMalloc(&d, 32)) return -2;
  cudaMemcpy(dc, hc, sizeof(IntCoef) * nc, cudaMemcpyHostToDevice);
  cudaMemcpy(dv, c, 8 * nc, cudaMemcpyHostToDevice);
  cudaMemcpy(ds, s, 8 * ns, cudaMemcpyHostToDevice);
  cudaMemset(d, 0, 32);
  check<<<1216, 256>>>(dc, dv, nc, ds, ns, pairs, d);
  const int rc = (int)cudaMemcpy(out, d, 32, cudaMemcpyDeviceToHost);
  cudaFree(dc); cudaFree(dv); cudaFree(ds); cudaFree(d);
  delete[] hc;
  return rc;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from foo_dsd_trellis_gb300 import build
    d = tmp_path_factory.mktemp("intmul")
    src, lib = d / "check.cu", d / "libcheck.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", build.CSRC,
                    "-I", os.path.join(build.ROOT, "include"), str(src), "-o", str(lib)], check=True)
    torch.cuda.init()
    L = C.CDLL(str(lib))

    def run(c, s, pairs):
        c, s = np.ascontiguousarray(c, np.float64), np.ascontiguousarray(s, np.float64)
        out = np.zeros(4, np.uint64)
        rc = L.run(C.c_void_p(c.ctypes.data), len(c), C.c_void_p(s.ctypes.data), C.c_longlong(len(s)), pairs,
                   C.c_void_p(out.ctypes.data))
        assert rc == 0
        return [int(v) for v in out]
    return run


def _doubles(exps, mants, signs=(0, 1)):
    b = np.array([(sg << 63) | (e << 52) | m for sg in signs for e in exps for m in mants], np.uint64)
    return b.view(np.float64)


def _mantissas(rng):
    full = (1 << 52) - 1
    m = [0, 1, 2, 3, full, full - 1, full - 2, 1 << 51, (1 << 51) - 1, (1 << 51) + 1, 0x5555555555555, 0xAAAAAAAAAAAAA,
         0xFFFFFFFF, 0x100000000, 0xFFFFF00000000, 0x6A09E667F3BCC, 0x6A09E667F3BCD]   # sqrt 2: on either side of 2^53
    m += [full ^ (full >> k) for k in range(1, 52, 3)] + [full >> k for k in range(1, 52, 3)]
    # 25 to 28 leading bits: products of about twice as many, exact ties among them
    m += [int(v) << (52 - k) for k in (25, 26, 27, 28) for v in rng.integers(0, 1 << k, 24)]
    m += [int(v) for v in rng.integers(0, 1 << 52, 40)]
    return sorted(set(m))


def test_built_operands(check):
    rng = np.random.default_rng(2)
    m = _mantissas(rng)
    c = _doubles((923, 924, 1022, 1023, 1024, 1122, 1123), m)
    s = np.concatenate([_doubles((200, 201, 1021, 1022, 1023, 1024, 1799, 1800), m), [0.0, -0.0]])
    n, bad, n0, bad0 = check(c, s, 0)
    assert n >= 2 * 7 * len(m) * 2 * 7 * len(m) and n0 == n + 2 * len(c)
    assert (bad, bad0) == (0, 0)


def test_random_operands(check):
    rng = np.random.default_rng(3)
    bits = lambda n, lo, hi: ((rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)) |
                              (rng.integers(lo, hi, n).astype(np.uint64) << np.uint64(52)) |
                              rng.integers(0, 1 << 52, n).astype(np.uint64)).view(np.float64)
    c, s = bits(997, 923, 1124), bits(1 << 23, 200, 1800)
    n, bad, n0, bad0 = check(c, s, 1)
    assert n == n0 == 1 << 23
    assert (bad, bad0) == (0, 0)


def test_out_of_range(check):
    """What has no integer form: range_word and range_word0 keep it out (the
    check kernel multiplies only what they let in)."""
    s = np.array([np.inf, -np.inf, np.nan, 5e-324, -1e-310, 2.0 ** -824, 1e300, -1e300, 0.0, -0.0])
    n, bad, n0, bad0 = check(np.array([0.75, -1.5]), s, 0)
    assert n == 0 and n0 == 4 and bad == bad0 == 0
