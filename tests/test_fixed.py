"""The fast mode's fixed-point rotation and sphere centres (csrc/af3d_fixed.cuh) on the host: no
further from the exact result (extended precision) than the FP64 formulas they stand in for, over
angles up to 2^-10 rad and coordinates from zero to hundreds of centimetres, and refused (left to
the FP64 formulas) outside their range."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avalancheflume3d_gb300", "csrc")

HOST = r"""
#include "af3d_fixed.cuh"
int af3d::g_estimate_ulps = 0;
extern "C" void run(const double *w, const double *R, const double *r, const double *pos, long n, int q, double *Rn,
                    double *s, int *ok) {
  for (long k = 0; k < n; k++) {
    long long t[9];
    ok[2 * k] = af3d::rotate_fixed(w + 3 * k, R + 9 * k, t);
    if (!ok[2 * k]) continue;
    for (int i = 0; i < 9; i++) Rn[9 * k + i] = af3d::double_of(t[i], 62);
    ok[2 * k + 1] = af3d::spheres_fixed(t, r + 3 * k, pos[k], q, s + 12 * k);
  }
}
"""
LD = np.longdouble
CORNERS = np.array(((1, 1, 1), (1, -1, -1), (-1, -1, 1), (-1, 1, -1)))


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    (d / "h.cpp").write_text(HOST)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-I", cuda + "/include", "-o",
                    str(d / "h.so"), str(d / "h.cpp")], check=True)
    lib = C.CDLL(str(d / "h.so"))

    def call(w, R, r, pos, q):
        n = len(w)
        Rn, s, ok = np.zeros((n, 3, 3)), np.zeros((n, 4, 3)), np.zeros((n, 2), dtype=np.int32)
        p = lambda a: np.ascontiguousarray(a).ctypes.data_as(C.c_void_p)
        lib.run(p(w), p(R), p(r), p(pos), C.c_long(n), q, p(Rn), p(s), p(ok))
        return Rn, s, ok.astype(bool)
    return call


def rotations(g, n):
    q = g.standard_normal((n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1)[:, None]).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                  1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                  1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)
    return R / np.sqrt((R * R).sum(1))[:, None]


def formulas(w, R, r, rad, T):
    """init_Verlet's rotation, renormalisation and sphere centres with the real type T."""
    w, R, r, rad = (a.astype(T) for a in (w, R, r, rad))
    t = (w * w).sum(1)
    A = 1 - t / 6 * (1 - t / 20 * (1 - t / 42))
    B = (1 - t / 12 * (1 - t / 30 * (1 - t / 56))) / 2
    x, y, z = w.T
    K = np.zeros(R.shape, dtype=T)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 0], K[:, 1, 2], K[:, 2, 0], K[:, 2, 1] = -z, y, z, -x, -y, x
    dR = A[:, None, None] * K + B[:, None, None] * w[:, :, None] * w[:, None, :]
    for i in range(3):
        dR[:, i, i] += 1 - t * B
    N = np.stack([sum(dR[:, i, k, None] * R[:, k] for k in range(3)) for i in range(3)], 1)
    N = N / np.sqrt((N * N).sum(1))[:, None]
    pos = rad / np.sqrt(T(2))
    s = np.stack([r + pos[:, None] * (N * c.astype(T)).sum(2) for c in CORNERS], 1)
    return N, s


@pytest.mark.parametrize("qs,scale", [(22, 1.0), (21, 1.2), (12, 1000.0), (29, 0.01)])
def test_no_further_off_than_fp64(run, qs, scale):
    g = np.random.default_rng(5)
    n = 60_000
    w = g.standard_normal((n, 3)) * 10.0 ** g.uniform(-9, -3.7, (n, 1))
    w[::50] = 0.0
    w[1::50, 1] = 0.0
    R = rotations(g, n)
    r = g.standard_normal((n, 3)) * np.array([120.0, 10.0, 1.0]) * 10.0 ** g.uniform(-3, 0, (n, 3)) * scale
    rad = g.uniform(0.05, 0.1, n) * scale
    Rn, s, ok = run(w, R, r, rad / np.sqrt(2.0), qs + 38)
    big = (np.abs(w) >= 2.0 ** -10).any(1) | ((w * w).sum(1) > 0.9 * 2.0 ** -20)
    assert ok[~big].all()
    k = ok.all(1)
    exact, one = formulas(w[k], R[k], r[k], rad[k], LD), formulas(w[k], R[k], r[k], rad[k], np.float64)
    # in units in the last place of a value, or of a thousandth of the scale (1, the spheres') below it
    for got, want, fp64, size in zip((Rn[k], s[k]), exact, one, (1.0, scale)):
        unit = np.spacing(np.maximum(np.abs(want).astype(np.float64), 1e-3 * size))
        err = lambda v: (np.abs(v.astype(LD) - want) / unit).astype(np.float64)
        mine, theirs = err(got), err(fp64)
        assert np.sqrt((mine ** 2).mean()) <= np.sqrt((theirs ** 2).mean())
        assert mine.max() <= theirs.max()


def test_refused_outside_the_range(run):
    g = np.random.default_rng(6)
    w, R = g.standard_normal((8, 3)) * 1e-5, rotations(g, 8)
    r, pos = np.zeros((8, 3)), np.full(8, 0.07)
    w[0, 1], w[1, 2], w[2, 0] = 2.0 ** -10, -1.0, np.nan
    R[3] *= 1.0 + 1e-8
    R[4, 0, 0] = np.inf
    r[5, 1], pos[6] = 1e300, 1e9
    _, _, ok = run(w, R, r, pos, 60)
    assert ok.tolist() == [[False, False]] * 5 + [[True, False]] * 2 + [[True, True]]
