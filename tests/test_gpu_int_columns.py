"""FP64 blocks of p = 3 and 4 (p = 2 on larger meshes) multiply most of each row's columns on the
integer pipe (step_body.cuh): exact products of the doubles' mantissas to 64
bits, summed in 128.

* K u on random, graded (each degree 1e-3 of the one below), near-constant, very
  large, very small, denormal and partly zero coefficients against sums of the
  exact products of the same blocks in extended precision.  Bar per row: the
  FP64 columns of a thread are summed in two chains of at most 12 terms per
  block, so with nb blocks the row is off by at most (12 nb + 16) 2^-53 of
  sum |K||u| (16: the chains', slices' and accumulators' own sums); the integer
  columns add less than 2^-60 of theirs.
* that error is no larger than twice what a plain FP64 sum makes, plus 4 ulp.
* infinities and NaN in any column still end in EXIT_INSTAB.
"""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import MatrixFree, _lib, mesh as M
from lymph3d_apsc_gb300._lib import LymphError

pytestmark = pytest.mark.gpu


def _solver(p, kind="bfs"):
    if kind == "tet":
        m = M.cube(2, bc="reference", agglomeration="tet", jitter=0.2)
    elif kind == "wide":   # a row of 17 blocks: a second batch of the gather
        m = M.cube(7, bc="reference", agglomeration="bfs", seed=1, group=(8, 100), jitter=0.15)
    else:
        # p = 2 takes this path from 608 polyhedra of long rows on
        m = M.cube(10 if p == 2 else 3, bc="reference", agglomeration="bfs", seed=1, group=(4, 12), jitter=0.15)
        m.mat, m.tet_mat = M.lognormal_materials(m.n_poly, seed=1), m.tet_poly.copy()
    g = MatrixFree(m, p, 1e-4)
    g.MAKE_MATRICES_FREE()
    return g


def _states(g, rng):
    deg = np.array([a + b + c for a in range(g.degree, -1, -1) for b in range(g.degree - a, -1, -1)
                    for c in range(g.degree - a - b, -1, -1)])
    u = rng.standard_normal((g.n_poly, 3, g.Np))
    smooth = 1e-12 * u
    smooth[:, :, deg == 0] += 1.0
    holes = u.copy()
    holes[::2] = 0.0
    holes[:, 1] = 0.0
    return {"random": u, "graded": u * 10.0 ** (-3.0 * deg), "smooth": smooth, "large": u * 1e250, "small": u * 1e-290,
            "denormal": u * 1e-310, "holes": holes, "graded up": u * 10.0 ** (3.0 * deg)}


@pytest.mark.parametrize("p,kind", [(2, "bfs"), (3, "tet"), (3, "bfs"), (3, "wide"), (4, "tet"), (4, "bfs"), (4, "wide")])
def test_operator_error_is_that_of_fp64(require_gpu, kind, p):
    g = _solver(p, kind)
    K, (rp, col) = g.blocks(), g.pattern()
    row = np.repeat(np.arange(g.n_poly), np.diff(rp))
    ext = np.longdouble
    for name, u in _states(g, np.random.default_rng(p)).items():
        u = u.reshape(g.n_poly, g.nd)
        got = g.apply_operator(u)
        k = -round(np.log2(np.abs(u).max()))              # sums in range for the reference
        us, gs = np.ldexp(u, k), np.ldexp(got, k)
        terms = K.astype(ext) * us[col][:, None, :].astype(ext)
        ref = np.zeros((g.n_poly, g.nd), ext)
        ab, fp64 = np.zeros((g.n_poly, g.nd)), np.zeros((g.n_poly, g.nd))
        np.add.at(ref, row, terms.sum(axis=2))
        np.add.at(ab, row, np.abs(terms).sum(axis=2).astype(np.float64))
        for b in range(len(col)):
            fp64[row[b]] += K[b] @ us[col[b]]
        tiny = np.ldexp(1.0, k - 1064)                    # a result below the normal range is rounded to it
        err = np.abs(gs - ref).astype(np.float64)
        plain = np.abs(fp64 - ref).astype(np.float64)
        nb = np.diff(rp)[:, None]
        assert (err <= (12 * nb + 16) * 2.0 ** -53 * ab + tiny).all(), name
        ok = ab > tiny * 2.0 ** 60
        if not ok.any():
            continue                                      # every row near the smallest double
        e, f = float((err[ok] / ab[ok]).max()), float((plain[ok] / ab[ok]).max())
        print(f"p={p} {kind} {name}: error / sum |K||u| {e:.2e}, plain FP64 {f:.2e}")
        assert e <= 2.0 * f + 4.0 * 2.0 ** -53, name
    g.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("column", [0, -1])
@pytest.mark.parametrize("p", [2, 3, 4])
def test_non_finite_states_are_reported(require_gpu, p, column, bad):
    g = _solver(p)
    u = np.random.default_rng(0).standard_normal((g.n_poly, g.nd))
    g.set_state(_lib.SLOT_U0, u)
    u[g.n_poly // 2, column] = bad
    g.set_state(_lib.SLOT_UN, u)
    with pytest.raises(LymphError) as e:
        g.TIME_STEP_MATRIX_FREE(g.dt)
    assert e.value.code == _lib.LYMPH_EXIT_INSTAB
    g.close()
