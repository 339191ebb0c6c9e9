"""A batched context whose meshes straddle the size from which a mesh gets launches of its own (32768 cells):
both kinds run as parallel branches and finish every step together. RK4 and RKDP54 against the oracle, FP64
1e-9 and mixed 1e-4 of Ms, at a fixed step; the step controller (rejected steps, error norm and torque maximum
carried by a large or a small mesh) in FP64; and the options of a large mesh against its per-mesh run."""
import numpy as np
import pytest

from oracle_libs import sphere_random, tilted_z, OracleSolver

pytestmark = pytest.mark.gpu

H = (4e-9, 4e-9, 3e-9)
# large with a Stockham y pass only (Ny 2048, 1536), and a large film without a register one (Ny 1536: work lists)
SIZES = {"mixed sizes": [(181, 182, 1), (64, 64, 8), (30, 20, 1), (48, 43, 16), (20, 24, 2)],
         "large only": [(256, 128, 1), (97, 85, 4)],
         "long lines": [(20, 1000, 2), (24, 700, 2), (47, 700, 1), (20, 24, 2)]}


def _desc(n, **kw):
    return dict(dict(n=n, h=H, Ms=8e5, A=1.3e-11, alpha=0.1, modules=1 | 2 | 16, Ha=(1e3, 0, 0)), **kw)


def _ctx(bm, descs, prec="fp64", batched=True):
    c = bm.Context(precision=bm.FP64 if prec == "fp64" else bm.MIXED)
    for q, d in enumerate(descs):
        c.add_mesh(d["n"], d["h"])
        c.set_material(q, Ms=d["Ms"], A=d["A"], alpha=d["alpha"], D=d.get("D", 0.0), K1=d.get("K1", 0.0))
        if "Ms_map" in d:
            c.set_material_maps(q, Ms_map=d["Ms_map"], K1_map=d["K1_map"])
        c.set_modules(q, d["modules"])
        c.set_field(q, d["Ha"])
        c.set_pbc(q, d.get("pbc", (0, 0, 0)))
    c.set_batched(batched)
    return c


@pytest.mark.parametrize("which", sorted(SIZES))
@pytest.mark.parametrize("ode", [0, 1])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
def test_batched_solo_meshes(bm, which, ode, prec, tol):
    descs = [_desc(n) for n in SIZES[which]]
    s = OracleSolver(descs, evaluation=ode, dt=2e-14, dT_min=2e-14, dT_max=2e-14)
    c = _ctx(bm, descs, prec)
    c.setode("RKDP54" if ode else "RK4", 2e-14)
    if ode:
        c.astepctrl(1e-4, 2.0, 2e-14, 2e-14)
    for q, d in enumerate(descs):
        M = sphere_random(int(np.prod(d["n"])), seed=3 + q, Ms=d["Ms"])
        s.set_m(M, q)
        c.set_m(M, q)
    c.get_mxh()
    s.get_mxh()
    s.run(5)
    st = c.run(5)
    assert st["accepted"] == 5 and abs(st["time"] - 1e-13) < 1e-24
    assert abs(c.get_mxh() / s.get_mxh() - 1) < (1e-9 if prec == "fp64" else 1e-4)
    err = max(np.abs(c.get_m(q) - s.get_m(q)).max() / d["Ms"] for q, d in enumerate(descs))
    c.close()
    s.close()
    assert err < tol


@pytest.mark.parametrize("hot", [0, 1, 2, 3])
def test_batched_solo_controller(bm, hot):
    """Adaptive RKDP54 with rejected steps: the mesh that starts in disorder carries the error norm and the torque
    maximum; counts, step, error norm, torque and states follow the oracle (FP64)."""
    descs = [_desc(n) for n in [(181, 182, 1), (64, 64, 8), (48, 43, 16), (20, 24, 2)]]
    ctrl = (1e-6, 2.0, 1e-15, 3e-12)
    s = OracleSolver(descs, evaluation=1, dt=2e-13, tol=ctrl[0], dT_incr=ctrl[1], dT_min=ctrl[2], dT_max=ctrl[3])
    c = _ctx(bm, descs)
    c.setode("RKDP54", 2e-13)
    c.astepctrl(*ctrl)
    for q, d in enumerate(descs):
        n = int(np.prod(d["n"]))
        M = sphere_random(n, seed=5 + q, Ms=d["Ms"]) if q == hot else tilted_z(n, seed=5 + q, max_deg=3.0, Ms=d["Ms"])
        s.set_m(M, q)
        c.set_m(M, q)
    c.get_mxh()
    s.get_mxh()
    so, sg = s.run(6), c.run(6)
    assert so["rejected"] >= 1
    assert sg["accepted"] == so["accepted"] and sg["rejected"] == so["rejected"]
    for k in ("time", "dT", "last_lte"):
        assert abs(sg[k] / so[k] - 1) < 1e-6, k
    assert abs(c.get_mxh() / s.get_mxh() - 1) < 1e-6
    err = max(np.abs(c.get_m(q) - s.get_m(q)).max() / d["Ms"] for q, d in enumerate(descs))
    c.close()
    s.close()
    assert err < 1e-8


@pytest.mark.parametrize("option", ["es RK4", "es RKDP54", "periodic", "maps", "idmi and anisotropy"])
def test_batched_solo_options(bm, option):
    """Evaluation speedup, periodic axes, material maps, iDMI and anisotropy of large meshes beside a small one:
    the batch follows the per-mesh run (FP64)."""
    kw = {"periodic": dict(pbc=(2, -1, 0)), "idmi and anisotropy": dict(modules=1 | 4 | 8 | 16, D=1.5e-3, K1=2e5)}.get(option, {})
    descs = [_desc(n, **kw) for n in [(181, 182, 1), (64, 64, 8), (20, 24, 2)]]
    if option == "maps":
        for q, d in enumerate(descs):
            rng = np.random.default_rng(q)
            n = int(np.prod(d["n"]))
            d.update(Ms_map=8e5 * rng.uniform(0.9, 1.1, n), K1_map=1e5 * rng.uniform(0.5, 1.5, n), modules=1 | 2 | 8 | 16)
    out = []
    for batched in (False, True):
        c = _ctx(bm, descs, batched=batched)
        c.setode("RKDP54" if option == "es RKDP54" else "RK4", 2e-14)
        if option == "es RKDP54":
            c.astepctrl(1e-5, 2.0, 1e-15, 3e-12)
        if option.startswith("es"):
            c.evalspeedup(2)
        for q, d in enumerate(descs):
            c.set_m(sphere_random(int(np.prod(d["n"])), seed=3 + q, Ms=d["Ms"]) * (d["Ms_map"][:, None] / d["Ms"] if "Ms_map" in d else 1), q)
        st = c.run(8)
        out.append((st["accepted"], st["rejected"], [c.get_m(q) / d["Ms"] for q, d in enumerate(descs)]))
        c.close()
    assert out[0][:2] == out[1][:2]
    assert max(np.abs(a - b).max() for a, b in zip(out[0][2], out[1][2])) < (1e-8 if option == "es RKDP54" else 1e-10)
