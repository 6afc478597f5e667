"""The integer-pipe FP64 division and square root (csrc/af3d_intfp64.cuh): equal to the correctly
rounded instructions bit for bit, on the host (with the FP32 estimates off by up to two units in
the last place either way) and on the device."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avalancheflume3d_gb300", "csrc")

HOST = r"""
#include "af3d_intfp64.cuh"
#include <cstddef>
int af3d::g_estimate_ulps = 0;
extern "C" void run(const double *a, const double *b, long n, int ulps, double *q, double *s) {
  af3d::g_estimate_ulps = ulps;
  for (long i = 0; i < n; i++) {
    q[i] = af3d::div_rn(a[i], b[i]);
    s[i] = af3d::sqrt_rn(a[i]);
  }
}
"""


def operands(n=200_000):
    """Pairs (a, b): random bit patterns of every exponent, moderate exponents with random, sparse
    and dense mantissas, quotients next to a rounding midpoint, squares and their neighbours, and
    the edges of the number line."""
    g = np.random.default_rng(11)
    bits = lambda m: g.integers(0, 1 << 63, m, dtype=np.uint64) << np.uint64(1) | g.integers(0, 2, m, dtype=np.uint64)
    any_a, any_b = bits(n).view(np.float64), bits(n).view(np.float64)
    mant = lambda m: (bits(m) & np.uint64(0x000FFFFFFFFFFFFF))
    make = lambda man: (man | (np.uint64(1023) + g.integers(-20, 20, len(man)).astype(np.int64).view(np.uint64))
                        << np.uint64(52)).view(np.float64)
    sparse = mant(n) & (~np.uint64(0) << g.integers(0, 52, n).astype(np.uint64))
    dense = mant(n) | ((np.uint64(1) << g.integers(0, 52, n).astype(np.uint64)) - np.uint64(1))
    a = [any_a, make(mant(n)), make(sparse), make(dense), make(mant(n))]
    b = [any_b, make(mant(n)), make(sparse[::-1].copy()), make(dense[::-1].copy()), make(sparse)]
    q = make(mant(n))
    near = b[1] * np.nextafter(q, np.inf) * 0.5 + b[1] * q * 0.5
    sq = q * q
    a += [near, sq, np.nextafter(sq, np.inf), np.nextafter(sq, 0)]
    b += [b[1], q, q, q]
    edge = np.array([0.0, -0.0, 1.0, 2.0, 3.0, 0.5, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** -1021,
                     np.finfo(np.float64).max, 2.0 - 2.0 ** -52, 1.0 - 2.0 ** -53, 4.0, -1.0, 1e-310, 2.0 ** 1023])
    a.append(np.repeat(edge, len(edge)))
    b.append(np.tile(edge, len(edge)))
    return np.concatenate(a), np.concatenate(b)


def same(x, y):
    return (x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1])
def test_host_build_is_correctly_rounded(tmp_path, ulps):
    src, so = tmp_path / "h.cpp", tmp_path / "h.so"
    src.write_text(HOST)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", CSRC, "-I", cuda + "/include",
                    "-o", str(so), str(src)], check=True)
    a, b = operands()
    q, s = np.empty_like(a), np.empty_like(a)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    C.CDLL(str(so)).run(p(a), p(b), C.c_long(len(a)), ulps, p(q), p(s))
    with np.errstate(all="ignore"):
        assert same(q, a / b).all()
        assert same(s, np.sqrt(a)).all()


@pytest.mark.gpu
def test_device_equals_the_instructions():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    a, b = operands(500_000)
    x = np.ascontiguousarray(np.concatenate([a, b[::-1]]))   # element i is divided by element n - 1 - i
    bad = np.zeros(len(x), dtype=np.int32)
    assert af3d.lib().af3d_check_fp64_bits(x.ctypes.data_as(C.c_void_p), len(x), bad.ctypes.data_as(C.c_void_p)) == 0
    assert not bad.any(), [(float(x[i]).hex(), float(x[-1 - i]).hex(), int(bad[i])) for i in np.nonzero(bad)[0][:10]]
