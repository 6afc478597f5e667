"""The integer-pipe division and square root (csrc/af3d_intfp64.cuh) with FP32 estimates off by up to three
units in the last place either way, also where that takes an estimate past 1 (divisors and squares just
above a power of two): correctly rounded."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from tests.test_intfp64 import CSRC, HOST, operands, same


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("intfp64")
    src, so = d / "h.cpp", d / "h.so"
    src.write_text(HOST)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", CSRC, "-I",
                    cuda + "/include", "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("ulps", [-3, -2, -1, 0, 1, 2, 3])
def test_any_estimate_within_three_ulps(host, ulps):
    a, b = operands(200_000)
    # mantissas at and just above one, where the estimate of the reciprocal (root) is one
    k = np.concatenate([np.arange(4096), 1 << np.arange(12, 45)]).astype(np.uint64)
    ones = (np.uint64(0x3FF0000000000000) + k).view(np.float64)
    num = np.random.default_rng(3).uniform(1.0, 2.0, len(ones))
    a, b = np.concatenate([a, num, ones, 4.0 * ones]), np.concatenate([b, ones, num, ones])
    q, s = np.empty_like(a), np.empty_like(a)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    host.run(p(a), p(b), C.c_long(len(a)), ulps, p(q), p(s))
    with np.errstate(all="ignore"):
        assert same(q, a / b).all()
        assert same(s, np.sqrt(a)).all()
