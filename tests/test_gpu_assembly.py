"""The FP64 block assembly from mass moments (k_assemble_self, k_assemble_nb)
at the forms the shared parity meshes do not reach: theta = 0 and 1, and a
polyhedron of 162 tetrahedra and 108 shared triangles (many rounds of the
tetrahedron and face tables).  Every block of K and A_dg against the oracle,
normwise <= 1e-12 over the mesh (the bar of the other set-up data: sums of at
most ~1e4 products of O(1) condition, eps * 1e4 = 2e-12 worst case, ~1e-14
expected), and M exactly symmetric.
"""
import math

import numpy as np
import pytest

from lymph3d_apsc_gb300 import MatrixFree, _lib, mesh as M
from oracle.oracle_py import Oracle
from test_gpu_mf import _big_polyhedron_mesh

pytestmark = pytest.mark.gpu


def _blocks_close(m, p, theta):
    o = Oracle(m, p, 1e-3, theta=theta)
    o.make_matrices()
    with MatrixFree(m, p, 1e-3, theta=theta) as g:
        g.MAKE_MATRICES_FREE()
        rp, col = g.pattern()
        for which in (_lib.BLOCKS_K, _lib.BLOCKS_ADG):
            vals, ref = g.blocks(which), o.block_dict(which)
            num = den = 0.0
            for P in range(g.n_poly):
                for k in range(rp[P], rp[P + 1]):
                    r = ref[(P, int(col[k]))]
                    num += float(np.sum((vals[k] - r) ** 2))
                    den += float(np.sum(r ** 2))
            assert math.sqrt(num / den) <= 1e-12, (which, math.sqrt(num / den))
        for which in (0, 1):
            mm = g.mass(which)
            assert np.array_equal(mm, mm.transpose(0, 2, 1))
    o.close()


@pytest.mark.parametrize("theta", [0.0, 1.0])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_blocks_of_other_penalty_forms(require_gpu, p, theta):
    m = M.cube(2, bc="reference", agglomeration="bfs", seed=3, group=(4, 12), jitter=0.2)
    mats = M.lognormal_materials(m.n_poly, seed=3)
    m.mat, m.tet_mat = mats, m.tet_poly.copy()
    _blocks_close(m, p, theta)


@pytest.mark.parametrize("p", [1, 2, 4])
def test_blocks_of_a_large_polyhedron(require_gpu, p):
    _blocks_close(_big_polyhedron_mesh(), p, -1.0)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_rhs_of_every_data_combination(require_gpu, p):
    """Every forcing / Dirichlet / Neumann id together (zero functions do no
    quadrature): normwise <= 1e-12 of the oracle's vector, exactly zero where
    all three are zero; projections of zero functions exactly zero."""
    m = M.cube(2, bc="reference", agglomeration="bfs", seed=5, group=(4, 12), jitter=0.2, material=(1.0, 2.0, 1.0))
    o = Oracle(m, p, 1e-3)
    o.make_matrices()
    with MatrixFree(m, p, 1e-3) as g:
        g.MAKE_MATRICES_FREE()
        for f in range(3):
            for d in range(3):
                for n in range(3):
                    g.MAKE_RHS_FREE(_lib.RHS_DYN, f, d, n)
                    o.make_rhs(1, f, d, n)
                    ref, got = o.rhs(1), g.rhs(_lib.RHS_DYN)
                    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref), (f, d, n)
        for fun in (_lib.FUN_IC_DISPLACEMENT, _lib.FUN_UEX_STAT):
            g.set_state(_lib.SLOT_UEX, np.ones((g.n_poly, g.nd)))
            g.COMPUTE_MODAL_COEFFICIENTS_FREE(fun, _lib.SLOT_UEX, 0.5)
            assert not g.get_state(_lib.SLOT_UEX).any()
    o.close()


@pytest.mark.parametrize("kind", ["one_poly", "tet_ref_jitter", "bfs_lognormal", "big"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_error_norms_of_rough_states(require_gpu, kind, p):
    """The DG norm by quadrature and the L2 norm, of random coefficients (no
    cancellation between the terms of the quadratic forms): 1e-11 relative of
    the oracle's assembled forms (block entries of ~1e4 rounded terms each,
    1e4 eps = 2e-12, and their mild cancellation in the forms)."""
    from test_gpu_parity import _mesh
    m = _big_polyhedron_mesh() if kind == "big" else _mesh(kind)
    o = Oracle(m, p, 1e-3)
    o.make_matrices()
    rng = np.random.default_rng(p)
    with MatrixFree(m, p, 1e-3) as g:
        g.MAKE_MATRICES_FREE()
        for slot in (_lib.SLOT_UN, _lib.SLOT_UEX):
            u = rng.standard_normal((g.n_poly, g.nd))
            g.set_state(slot, u)
            o.set_state(slot, u)
        for got, ref in ((g.COMPUTE_ERROR_L2_MATRIX_FREE(), o.error_l2(1, 3)), (g.COMPUTE_ERROR_DG_MATRIX_FREE(), o.error_dg(1, 3))):
            assert abs(got - ref) <= 1e-11 * abs(ref), (got, ref)
    o.close()


@pytest.mark.parametrize("p", [1, 4])
def test_geometry_of_a_large_polyhedron(require_gpu, p):
    """Boxes and diameters (a polyhedron of 648 vertex entries reads them from
    device memory): the oracle's boxes, diameters to the last bit or two."""
    m = _big_polyhedron_mesh()
    o = Oracle(m, p, 1e-3)
    with MatrixFree(m, p, 1e-3) as g:
        (bb, hk), (rb, rk) = g.poly_geometry(), o.poly_geometry()
        assert np.array_equal(bb, rb)
        assert np.abs(hk / rk - 1.0).max() <= 1e-15
    o.close()
