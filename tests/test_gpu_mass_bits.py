"""The mass matrices keep the reference's operations and their order (setup.cu), the
divisions by an interval's constants included, which div_known forms in two operations:
entries a <= b, which the factorisation reads, equal the oracle's bit for bit (a quotient's
sum before its one rounding is off by 2^-105: fewer than one entry in 2^40 could differ)."""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import MatrixFree, _lib, mesh as M
from oracle.oracle_py import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED, _lib.MIXED_MF])
@pytest.mark.parametrize("agglomeration", ["bfs", "tet"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_mass_matrices_have_the_oracles_bits(require_gpu, p, agglomeration, precision):
    m = M.cube(3, bc="reference", agglomeration=agglomeration, seed=1, group=(4, 12), jitter=0.2)
    m.mat, m.tet_mat = M.lognormal_materials(m.n_poly, seed=1), m.tet_poly.copy()
    m.mat[:, 0] = np.random.default_rng(0).uniform(0.5, 2.0, len(m.mat))
    g = MatrixFree(m, p, 1e-3, precision=precision)
    g.MAKE_MATRICES_FREE()
    o = Oracle(m, p, 1e-3)
    o.make_matrices()
    up = np.triu_indices(g.Np)
    for which in (0, 1):
        got, ref = g.mass(which), np.asarray(o.mass(which)).reshape(-1, g.Np, g.Np)
        assert np.array_equal(got[:, up[0], up[1]], ref[:, up[0], up[1]])
        assert np.array_equal(got, got.transpose(0, 2, 1))
    g.close()
    o.close()
