"""A batched context whose meshes straddle the size from which a mesh gets launches of its own (32768 cells):
both kinds run as parallel branches and finish every step together. RK4 and RKDP54 against the oracle, FP64
1e-9 and mixed 1e-4 of Ms, at a fixed step, and the step statistics of the set."""
import numpy as np
import pytest

from oracle_libs import sphere_random, OracleSolver

pytestmark = pytest.mark.gpu

SIZES = {"mixed sizes": [(181, 182, 1), (64, 64, 8), (30, 20, 1), (48, 43, 16), (20, 24, 2)],
         "large only": [(256, 128, 1), (97, 85, 4)]}


@pytest.mark.parametrize("which", sorted(SIZES))
@pytest.mark.parametrize("ode", [0, 1])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
def test_batched_solo_meshes(bm, which, ode, prec, tol):
    descs = [dict(n=n, h=(4e-9, 4e-9, 3e-9), Ms=8e5, A=1.3e-11, alpha=0.1, modules=1 | 2 | 16, Ha=(1e3, 0, 0))
             for n in SIZES[which]]
    s = OracleSolver(descs, evaluation=ode, dt=2e-14, dT_min=2e-14, dT_max=2e-14)
    c = bm.Context(precision=bm.FP64 if prec == "fp64" else bm.MIXED)
    for q, d in enumerate(descs):
        c.add_mesh(d["n"], d["h"])
        c.set_material(q, Ms=d["Ms"], A=d["A"], alpha=d["alpha"])
        c.set_modules(q, d["modules"])
        c.set_field(q, d["Ha"])
    c.set_batched(True)
    c.setode("RKDP54" if ode else "RK4", 2e-14)
    if ode:
        c.astepctrl(1e-4, 2.0, 2e-14, 2e-14)
    for q, d in enumerate(descs):
        M = sphere_random(int(np.prod(d["n"])), seed=3 + q, Ms=d["Ms"])
        s.set_m(M, q)
        c.set_m(M, q)
    c.get_mxh()
    s.run(5)
    st = c.run(5)
    assert st["accepted"] == 5 and abs(st["time"] - 1e-13) < 1e-24
    assert c.get_mxh() > 0
    err = max(np.abs(c.get_m(q) - s.get_m(q)).max() / d["Ms"] for q, d in enumerate(descs))
    c.close()
    s.close()
    assert err < tol
