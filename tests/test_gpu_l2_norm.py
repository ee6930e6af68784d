"""The L2 norm's per-polyhedron sums, 10 / 4 / 2 / 1 polyhedra to a CTA at p = 1..4: whole
CTAs and remainders (1 to 162 polyhedra), against du^T M du from the
mass matrices read back (each sum of 3 Np Np products rounds by less than
(Np + 3 Np + 4) 2^-53 of its terms' sizes; numpy's own order as much again), and the
allocation-free entry point's bits."""
from ctypes import byref, c_double

import numpy as np
import pytest

from lymph3d_apsc_gb300 import MatrixFree, _lib, mesh as M
from test_zz_no_alloc import DeviceArray, _cudart

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [dict(n=1, agglomeration="hex"), dict(n=1, agglomeration="tet"), dict(n=2, agglomeration="hex"),
                                  dict(n=3, agglomeration="hex"), dict(n=2, agglomeration="bfs", group=(8, 40), seed=2),
                                  dict(n=3, agglomeration="tet")])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_l2_error(require_gpu, p, mesh):
    g = MatrixFree(M.cube(bc="reference", jitter=0.1, **mesh), p, 1e-3)
    g.MAKE_MATRICES_FREE()
    rng = np.random.default_rng(p)
    uh, uex = rng.standard_normal((2, g.n_poly, g.nd))
    g.set_state(_lib.SLOT_UN, uh)
    g.set_state(_lib.SLOT_UEX, uex)
    got = g.COMPUTE_ERROR_L2_MATRIX_FREE(_lib.SLOT_UN, _lib.SLOT_UEX)
    Mm = g.mass(1)
    du = (uh - uex).reshape(g.n_poly, 3, g.Np)
    ref = np.einsum("pir,prc,pic->", du, Mm, du)
    size = np.einsum("pir,prc,pic->", abs(du), abs(Mm), abs(du))
    assert abs(got - ref) <= 2 * (4 * g.Np + 4 + g.n_poly) * 2.0 ** -53 * size
    rt = _cudart()
    arr = [DeviceArray(rt, a) for a in (Mm, uh, uex)]
    out = c_double()
    assert g.lib.lymph_error_l2_noalloc(*[a.ptr for a in arr], g.n_poly, g.Np, byref(out)) == 0
    assert out.value == got
    for a in arr:
        a.free()
    g.close()
