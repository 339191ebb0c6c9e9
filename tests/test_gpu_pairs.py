"""Kernels that carry two x-adjacent values per thread, on cuda:0 against the oracle: the stage kernel's
per-cell part on cell pairs (even and odd nx down to 1, every field term, open and periodic, each x
transform variant at lengths that have it, the FP32 x transforms on butterfly pairs) and the FP32 z pass on
column pairs (BM_Z_XV=2; each length, partial tiles).
Bounds as elsewhere: FP64 1e-9 and mixed 1e-5 of the largest field, states FP64 1e-9, mixed 1e-4 of Ms."""
import numpy as np
import pytest

from oracle_libs import orc_hdemag, sphere_random, OracleSolver

pytestmark = pytest.mark.gpu
MU0 = 1.256637061435916e-6


# (x-transform variant, nx): every nx has the two-level / generic form; Stockham from 16 packed elements, radix 16
# at 256, 512 and 1024 of them
XV_NX = [("0", n) for n in (1, 2, 3, 16, 31, 190, 257)] + [("1", n) for n in (16, 31, 190, 257)] + \
        [("2", n) for n in (201, 256, 401, 512)]


@pytest.mark.parametrize("xv,nx", XV_NX)
@pytest.mark.parametrize("pbc", [(0, 0, 0), (2, -1, 1)])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
def test_stage_pairs(bm, monkeypatch, nx, pbc, xv, prec, tol):
    monkeypatch.setenv("BM_TILES", "1,1,4,2")
    monkeypatch.setenv("BM_STAGE_XV", xv)
    d = dict(n=(nx, 5, 3), h=(4e-9, 3e-9, 2e-9), Ms=8e5, A=1.3e-11, D=1.5e-3, alpha=0.1, K1=1e5, K2=2e4, ea=(0.3, 0.2, 0.9),
             modules=1 | 4 | 8 | 16, Ha=(2e4, -1e4, 5e3), pbc=pbc)
    M = sphere_random(int(np.prod(d["n"])), seed=9 + nx, Ms=8e5)
    # RKDP54 at a fixed step (dT_min = dT_max): adaptive steps scale with (error estimate)^(-1/6), so a
    # mixed-precision estimate at its rounding floor would compare states at different times
    for ode in (0, 1):
        s = OracleSolver([d], evaluation=ode, dt=2e-14, dT_min=2e-14, dT_max=2e-14)
        s.set_m(M)
        with bm.Context(precision=bm.FP64 if prec == "fp64" else bm.MIXED) as c:
            c.add_mesh(d["n"], d["h"])
            c.set_material(0, Ms=d["Ms"], A=d["A"], alpha=d["alpha"], K1=d["K1"], K2=d["K2"], ea=d["ea"], D=d["D"])
            c.set_modules(0, d["modules"])
            c.set_pbc(0, pbc)
            c.set_field(0, d["Ha"])
            c.setode("RKDP54" if ode else "RK4", 2e-14)
            if ode:
                c.astepctrl(1e-4, 2.0, 2e-14, 2e-14)
            c.set_m(M)
            H, Href = c.update_field(), s.heff()
            assert c.tiles()["stage_xv"] == int(xv)
            assert np.abs(H - Href).max() / np.abs(Href).max() < (1e-9 if prec == "fp64" else 1e-5)
            c.run(6)
            s.run(6)
            assert np.abs(c.get_m() - s.get_m()).max() / 8e5 < tol
        s.close()


@pytest.mark.parametrize("nx", [49, 64, 100, 128, 201, 256, 401, 512, 1000])
@pytest.mark.parametrize("rows", [1, 3])
@pytest.mark.parametrize("pbc", [(0, 0, 0), (2, -1, 1)])
def test_stage_butterfly_pairs(bm, monkeypatch, nx, rows, pbc):
    """The FP32 x transforms on butterfly pairs (BM_STAGE_XV=4), open and periodic, uniform and with Ms / K1 maps
    (three rows): field, RK4 and RKDP54 steps."""
    monkeypatch.setenv("BM_TILES", "1,1,4,%d" % (rows if nx < 600 else min(rows, 2)))
    monkeypatch.setenv("BM_STAGE_XV", "4")
    d = dict(n=(nx, 3, 2), h=(4e-9, 3e-9, 2e-9), Ms=8e5, A=1.3e-11, D=1.5e-3, alpha=0.1, K1=1e5, modules=1 | 4 | 8 | 16,
             Ha=(2e4, -1e4, 5e3), pbc=pbc)
    M = sphere_random(int(np.prod(d["n"])), seed=9 + nx, Ms=8e5)
    if rows == 3:
        rng = np.random.default_rng(nx)
        d["Ms_map"] = 8e5 * rng.uniform(0.9, 1.1, len(M))
        d["K1_map"] = 1e5 * rng.uniform(0.5, 1.5, len(M))
        M *= d["Ms_map"][:, None] / 8e5
    for ode in (0, 1):
        s = OracleSolver([d], evaluation=ode, dt=2e-14, dT_min=2e-14, dT_max=2e-14)
        s.set_m(M)
        with bm.Context(precision=bm.MIXED) as c:
            c.add_mesh(d["n"], d["h"])
            c.set_material(0, Ms=d["Ms"], A=d["A"], alpha=d["alpha"], K1=d["K1"], D=d["D"])
            if rows == 3:
                c.set_material_maps(0, Ms_map=d["Ms_map"], K1_map=d["K1_map"])
            c.set_modules(0, d["modules"])
            c.set_pbc(0, pbc)
            c.set_field(0, d["Ha"])
            c.setode("RKDP54" if ode else "RK4", 2e-14)
            if ode:
                c.astepctrl(1e-4, 2.0, 2e-14, 2e-14)
            c.set_m(M)
            if not any(pbc):
                H, Href = c.demag_field(), orc_hdemag(M, d["n"], d["h"])[0]
                assert np.abs(H - Href).max() / np.abs(Href).max() < 1e-5
            H, Href = c.update_field(), s.heff()
            assert c.tiles()["stage_xv"] == 4
            assert np.abs(H - Href).max() / np.abs(Href).max() < 1e-5
            c.run(6)
            s.run(6)
            assert np.abs(c.get_m() - s.get_m()).max() / 8e5 < 1e-4
        s.close()


@pytest.mark.parametrize("n,W", [((30, 7, 2), 8), ((16, 9, 3), 16), ((47, 6, 4), 32), ((100, 5, 6), 64), ((24, 12, 8), 16),
                                 ((33, 8, 11), 8), ((64, 16, 13), 32), ((5, 4, 16), 8), ((128, 3, 9), 32)])
def test_zpair_hdemag(bm, monkeypatch, n, W):
    monkeypatch.setenv("BM_TILES", "1,1,%d,1" % W)
    monkeypatch.setenv("BM_Z_XV", "2")
    h = (3e-9, 2e-9, 2.5e-9)
    M = sphere_random(int(np.prod(n)), seed=70 + n[0], Ms=8e5)
    Href, _ = orc_hdemag(M, n, h)
    with bm.Context(precision=bm.MIXED) as c:
        c.add_mesh(n, h)
        c.set_modules(0, bm.DEMAG)
        c.set_m(M)
        H = c.demag_field()
        assert c.tiles()["zmid_zv"] == 2 and c.tiles()["zmid_W"] == W
    assert np.abs(H - Href).max() / np.abs(Href).max() < 1e-5


@pytest.mark.parametrize("n", [(64, 5, 3), (33, 4, 3), (1, 6, 4), (2, 2, 2), (50, 1, 1), (7, 9, 1)])
@pytest.mark.parametrize("pbc", [(0, 0, 0), (1, 0, -1)])
@pytest.mark.parametrize("D", [0.0, 5e-6])
def test_stage_pairs_smooth_state(bm, n, pbc, D):
    """FP32 exchange / iDMI of a state that varies little from cell to cell, at every cell, the boundaries
    included. Differences of neighbours are exact there, so the error is bounded by the roundings after them:
    at most 20 (the boundary term 4, 1 / h^2, the sums over sides and axes 4, the coefficient 7, its product
    and the sum into H 2, the gradient's factors 2), each 2^-24 of the terms. A stencil that rounds a sum of two
    neighbours first is off by 2^-24 of M instead, a thousand times the differences here."""
    h, Ms, A = (4e-9, 3e-9, 2e-9), 8e5, 1.3e-11
    z, y, x = np.meshgrid(*[(np.arange(k) + 0.5) / k for k in n[::-1]], indexing="ij")
    th, ph = 0.9 + 3e-3 * np.cos(2 * x + y) + 2e-3 * z, 0.7 + 4e-3 * np.sin(x - 2 * y) - 2e-3 * z
    M = (Ms * np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], -1)).astype(np.float32).astype(np.float64)
    # terms of the stencil per cell: |neighbour - cell| per side, |h bd| at an open side
    rr = D / (2 * A)
    bd = {0: np.stack([rr * M[..., 2], 0 * M[..., 0], -rr * M[..., 0]], -1), 1: np.stack([0 * M[..., 0], rr * M[..., 2], -rr * M[..., 1]], -1),
          2: 0 * M}
    terms, grad = np.zeros_like(M), {}
    for k, ax in ((0, 2), (1, 1), (2, 0)):
        if n[k] == 1:
            continue
        d = np.abs(np.diff(M, axis=ax))
        lo, hi = [np.abs(h[k] * np.take(bd[k], [i], axis=ax)) for i in (0, -1)]
        if pbc[k]:
            wrap = np.abs(pbc[k] * np.take(M, [-1], axis=ax) - np.take(M, [0], axis=ax))
            lo = hi = wrap
        t = np.concatenate([lo, d], axis=ax) + np.concatenate([d, hi], axis=ax)
        terms += 2 * A / (MU0 * Ms * Ms) * t / h[k] ** 2
        grad[k] = D / (MU0 * Ms * Ms) * t / h[k]
    if 0 in grad:
        terms[..., 0] += grad[0][..., 2]
        terms[..., 2] += grad[0][..., 0]
    if 1 in grad:
        terms[..., 1] += grad[1][..., 2]
        terms[..., 2] += grad[1][..., 1]
    d = dict(n=n, h=h, Ms=Ms, A=A, D=D, modules=4 if D else 2, pbc=pbc)
    s = OracleSolver([d])
    s.set_m(M.reshape(-1, 3))
    Href = s.heff()
    s.close()
    with bm.Context(precision=bm.MIXED) as c:
        c.add_mesh(n, h)
        c.set_material(0, Ms=Ms, A=A, D=D, alpha=0.1)
        c.set_modules(0, d["modules"])
        c.set_pbc(0, pbc)
        c.set_m(M.reshape(-1, 3))
        H = c.update_field()
    bound = 20 * 2.0 ** -24 * terms.reshape(-1, 3) + 1e-9   # A/m; M and H are of the order of 1e5
    assert (np.abs(H - Href) <= bound).all()
