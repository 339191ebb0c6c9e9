"""The multilayered z pass on whole vectors per thread (BM_ML_W with BM_ML_VEC=1) on cuda:0 against the
oracle: H_demag FP64 1e-9 and mixed 1e-5 of max |H_ref| for two to eight layers, 2D (Nz = 1) and 3D common
grids of 2 to 4 planes (Nz = 4, 6, 8), equal and unequal cells (self, z-shifted and reused kernels), tile
widths that do not divide the row, block sizes that are not a multiple of a warp."""
import numpy as np
import pytest

from oracle_libs import MultiLayer, sphere_random
from test_gpu_ml import _ctx, _split, _relmax, NM
from test_oracle_ml import STACK3, WIDE_IRR

pytestmark = pytest.mark.gpu

EQUAL = [((24, 18, 1), (2 * NM, 2 * NM, 1 * NM), (0, 0, z * NM)) for z in (0, 2, 4, 7, 9, 11, 13, 16)]
CASES = [(STACK3, 0, None, 8), (STACK3, 0, None, 16), (STACK3, 2, None, 8), (STACK3, 1, None, 16), (WIDE_IRR, 0, None, 16),
         (STACK3, 0, (8, 8, 3), 8), (STACK3, 0, (8, 8, 4), 8), (EQUAL[:2], 0, None, 16), (EQUAL[:3], 0, None, 8), (EQUAL, 0, None, 8)]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("q", range(len(CASES)))
def test_ml_vec_hdemag(bm, monkeypatch, q, prec):
    meshes, mode, nc, W = CASES[q]
    monkeypatch.setenv("BM_ML_W", str(W))
    M = sphere_random(sum(int(np.prod(m[0])) for m in meshes), seed=21 + q, Ms=8e5)
    Href = MultiLayer(meshes, mode, nc).eval(M)
    H = {}
    for vec in ("0", "1"):
        monkeypatch.setenv("BM_ML_VEC", vec)
        with _ctx(bm, meshes, mode, nc, prec) as c:
            for i, Mi in enumerate(_split(M, meshes)):
                c.set_m(Mi, i)
            H[vec] = np.concatenate([c.demag_field(i) for i in range(len(meshes))])
    assert _relmax(H["1"], Href) < (1e-9 if prec == "fp64" else 1e-5)
    assert _relmax(H["1"], H["0"]) < (1e-13 if prec == "fp64" else 2e-6)   # two orders of the same products
