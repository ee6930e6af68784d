"""The integer columns of p = 2 (608 polyhedra or more, 8 blocks a row or more) on rows
longer than one batch of the gather (16 blocks): the second batch restarts the exponent
and the 128-bit sum.  Inputs, reference and bars are test_gpu_int_columns.py's."""
import numpy as np
import pytest

import test_gpu_int_columns as T
from lymph3d_apsc_gb300 import MatrixFree, mesh as M

pytestmark = pytest.mark.gpu


def _solver(p, kind):
    m = M.cube(12, bc="reference", agglomeration="bfs", seed=1, group=(4, 24), jitter=0.15)
    m.mat, m.tet_mat = M.lognormal_materials(m.n_poly, seed=1), m.tet_poly.copy()
    g = MatrixFree(m, p, 1e-4)
    g.MAKE_MATRICES_FREE()
    rp, _ = g.pattern()
    assert g.n_poly >= 608 and np.diff(rp).mean() >= 8 and np.diff(rp).max() > 16
    return g


def test_operator_error_is_that_of_fp64_on_long_rows(require_gpu, monkeypatch):
    monkeypatch.setattr(T, "_solver", _solver)
    T.test_operator_error_is_that_of_fp64(True, "long", 2)
