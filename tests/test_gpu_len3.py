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
