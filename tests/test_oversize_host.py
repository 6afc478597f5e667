"""af3d_step_host with clumps larger than the near lists reach for (csrc/af3d_near.cu), which make
every clump search its cells: the call equals import, step and export on a second context, byte for
byte.  The large clumps are the last of the array, so their lists are among the last to be built while
the force pass of the first part, which holds their partners, already runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


def corner_to(axis):
    """Rotation that takes the corner (1, 1, 1) / sqrt 3 of a clump to the unit vector `axis`."""
    a, b = np.full(3, 1.0 / np.sqrt(3.0)), np.asarray(axis, dtype=float)
    v, c = np.cross(a, b), float(a @ b)
    k = np.array([[0.0, -v[2], v[1]], [v[2], 0.0, -v[0]], [-v[1], v[0], 0.0]])
    return np.eye(3) + k + k @ k / (1.0 + c)


def pairs(af3d, n, scale):
    """n / 2 clumps of rmax in the air, each touching one of scale rmax from the end of the array: a
    sphere of each on the line between them, which runs along y."""
    from tests.states import flume_system, wall_state
    sys, fun = flume_system(n, time=0.0)
    pp = wall_state(n, 5, sys, vel=0.0, omega=0.0)
    rmax = float(sys["rmax"])
    m = n // 2
    big = np.arange(n - 1, n - 1 - m, -1)
    pp["radius"][big] = scale * rmax
    from oracle.pyoracle import GYR, mass_inertia, rotate_slope
    mass_inertia(pp)
    k = np.arange(m)
    gap = 0.5 * GYR * (1.0 + scale) * rmax - 0.02 * rmax
    pitch = 2.0 * gap
    # (columns shifted against each other, so that every distance to a cell border occurs)
    at = np.stack([60.0 + pitch * (k % 16), 8.0 + 1.37 * pitch * (k // 16 % 12) + 0.06 * (k % 16),
                   90.0 + pitch * (k // 192)], 1)
    pp["rr"][:m] = at
    pp["rr"][big] = at + np.array([0.0, gap, 0.0])
    for who, axis in ((np.arange(m), (0.0, 1.0, 0.0)), (big, (0.0, -1.0, 0.0))):
        R = corner_to(axis)
        for row, f in zip(R, ("Rmatx", "Rmaty", "Rmatz")):
            pp[f][who] = row
    af3d.sphere_centres(pp)
    rotate_slope(pp, sys)
    return sys, fun, pp


def coarse_grid(g):
    """The grid g with cells of twice the side."""
    g = g.copy()
    g["ncell"] = (g["ncell"] + 1) // 2
    g["cell_side"] *= 2.0
    g["cs_inv"] = 1.0 / g["cell_side"]
    g["rr_max"] = g["rr_min"] + g["ncell"] * g["cell_side"]
    g["length"] = g["rr_max"] - g["rr_min"]
    g["ncell3"] = int(np.prod(g["ncell"]))
    g["ntot"] = g["ncell3"] * g["ntags"]
    return g


@pytest.mark.parametrize("scale", [1.04, 1.06, 1.5])
@pytest.mark.parametrize("n", [3072, 9001])
def test_step_host_finds_oversize_partners(af3d, n, scale):
    sys, fun, pp0 = pairs(af3d, n, scale)
    with af3d.Engine(sys, fun, ntags=0) as a, af3d.Engine(sys, fun, ntags=0) as b:
        for e in (a, b):   # past the re-grid after the first step, then a grid of wide cells
            e.import_particles(pp0)
            e.step(1)
            e.set_grid(coarse_grid(e.get_grid()))
        pa, aa, la = pp0.copy(), np.zeros((n, 3)), np.zeros((n, 3))
        pb, ab, lb = pp0.copy(), aa.copy(), la.copy()
        for _ in range(3):
            a.contact_count()
            a.import_particles(pa, aa, la)
            a.step(1)
            assert a.contact_count() >= n // 2   # every pair touches
            pa, aa, la = a.export_particles()
            b.step_host(pb, ab, lb, acc_out=ab, anga_out=lb)
            assert pb.tobytes() == pa.tobytes()
            assert ab.tobytes() == aa.tobytes()
            assert lb.tobytes() == la.tobytes()
