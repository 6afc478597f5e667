"""Writes fast_device.npz: runs of the fast FP64 mode under the device friction law, as commit d99b290
computed them on a GB300 (python -m tests.runs.make_fast_device on that commit's tree).

Under that law every pushing pair slides in the Coulomb branch, and its direction v_t / |v_t| shows a
last-bit difference divided by the slip, so the runs are kept bit for bit.  One count per shape of the
force pass (up to 20,480 clumps and more), a filling pile and an ensemble; every stride-th clump."""
from __future__ import annotations

import pathlib

import numpy as np

PATH = pathlib.Path(__file__).with_name("fast_device.npz")
FIELDS = ("rr", "vv", "ww", "Rmatx", "Rmaty", "Rmatz", "rr_s")
# name: clumps (flumes of an ensemble), steps, stride of the stored clumps
RUNS = {"bed": (1409, 90, 16), "bed_large": (24001, 30, 256), "fill": (901, 40, 16), "ensemble": (3, 30, 512)}


def state(name):
    """(system_par, Funnel, particles, phase, ntags): a bed sheared downslope, a settling pile."""
    import avalancheflume3d_gb300 as af3d
    from avalancheflume3d_gb300.workloads import ensemble_configs, ensemble_state, flume_2k, flume_state
    n = RUNS[name][0]
    rng = np.random.default_rng(17)
    phase = af3d.PHASE_AVALANCHE
    if name == "ensemble":
        sys, fun, pp = ensemble_state(ensemble_configs(n, layout="bed", overlap=2.0e-5))
        cost, sint = (np.repeat(sys[k], sys["npart"]) for k in ("cost", "sint"))
    else:
        sys, fun, pp = flume_state(flume_2k(n=n, width=4.0, Lflume=80.0, overlap=2.0e-5,
                                            layout="pile" if name == "fill" else "bed"))
        cost, sint = float(sys["cost"]), float(sys["sint"])
    if name == "fill":
        phase = af3d.PHASE_FILL
        sys["time"] = -1.0
        sys["side"][0] = 15.0
        pp["vv"][:, 2] = -15.0
    else:
        z = pp["rrot"][:, 2]
        u = 110.0 * (0.5 + 0.5 * z / float(z.max()))
        pp["vv"][:, 0] = u * cost
        pp["vv"][:, 2] = -u * sint
    pp["vv"] += 4.0 * rng.standard_normal((len(pp), 3))
    pp["ww"] = 30.0 * rng.standard_normal((len(pp), 3))
    return sys, fun, pp, phase


def run(name):
    """{field: values of the stored clumps} after the run's steps."""
    import avalancheflume3d_gb300 as af3d
    sys, fun, pp, phase = state(name)
    _, steps, stride = RUNS[name]
    with af3d.Engine(sys, fun, phase=phase, friction=af3d.FRICTION_DEV, fp_mode=af3d.FP_FAST) as e:
        e.import_particles(pp)
        e.forces()
        e.swap_accel()
        e.step(steps)
        p, a, al = e.export_particles()
    out = {f: p[f] for f in FIELDS}
    out.update(a=a, alpha=al)
    return {f: np.ascontiguousarray(x[::stride]) for f, x in out.items()}


if __name__ == "__main__":
    np.savez_compressed(PATH, **{"%s_%s" % (name, f): x for name in RUNS for f, x in run(name).items()})
