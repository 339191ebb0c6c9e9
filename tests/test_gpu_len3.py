"""The two-level register y transforms of 3 * 2^k lengths (Ny 12 .. 768), 2D pass, 3D passes and the
batched 2D launch that mixes them, on cuda:0 against the oracle: H_demag FP64 1e-9 and mixed 1e-5 of
max |H_ref|, odd row counts and column counts that are not a multiple of the tile width."""
import numpy as np
import pytest

from oracle_libs import orc_hdemag, sphere_random, OracleSolver

pytestmark = pytest.mark.gpu

ROWS = [5, 11, 23, 48, 95, 190, 383]   # Ny = 12, 24, 48, 96, 192, 384, 768


@pytest.mark.parametrize("ny", ROWS)
@pytest.mark.parametrize("nz,W", [(1, 1), (1, 2), (3, 4)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_len3_hdemag(bm, monkeypatch, ny, nz, W, prec):
    monkeypatch.setenv("BM_TILES", "%d,%d,8,1" % (W, W))
    n, h = (11, ny, nz), (3e-9, 2e-9, 2.5e-9)
    M = sphere_random(int(np.prod(n)), seed=40 + ny, Ms=8e5)
    Href, _ = orc_hdemag(M, n, h)
    with bm.Context(precision=bm.FP64 if prec == "fp64" else bm.MIXED) as c:
        c.add_mesh(n, h)
        c.set_modules(0, bm.DEMAG)
        c.set_m(M)
        H = c.demag_field()
        assert c.tiles()["ypass_yv"] == 0
    assert np.abs(H - Href).max() / np.abs(Href).max() < (1e-9 if prec == "fp64" else 1e-5)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
@pytest.mark.parametrize("ode", [0, 1])
def test_len3_batched_branches(bm, prec, tol, ode):
    """Uneven films whose launches run as parallel branches; the step ends with the last item of them."""
    descs = [dict(n=n, h=(4e-9, 4e-9, 3e-9), Ms=8e5, A=1.3e-11, alpha=0.1, modules=1 | 2 | 16, Ha=(1e3, 0, 0))
             for n in ((17, 5, 1), (40, 11, 1), (24, 23, 1), (64, 48, 1), (33, 60, 1), (20, 24, 2), (70, 30, 4))]
    M0 = [sphere_random(int(np.prod(d["n"])), seed=3 + q, Ms=d["Ms"]) for q, d in enumerate(descs)]
    s = OracleSolver(descs, evaluation=ode, dt=2e-14)
    c = bm.Context(precision=bm.FP64 if prec == "fp64" else bm.MIXED)
    for q, d in enumerate(descs):
        c.add_mesh(d["n"], d["h"])
        c.set_material(q, Ms=d["Ms"], A=d["A"], alpha=d["alpha"])
        c.set_modules(q, d["modules"])
        c.set_field(q, d["Ha"])
    c.set_batched(True)
    c.setode("RKDP54" if ode else "RK4", 2e-14)
    for q, M in enumerate(M0):
        s.set_m(M, q)
        c.set_m(M, q)
    s.run(12)
    st = c.run(12)
    assert st["accepted"] == 12
    err = max(np.abs(c.get_m(q) - s.get_m(q)).max() / d["Ms"] for q, d in enumerate(descs))
    c.close()
    s.close()
    assert err < tol
