"""A batch equals its problems stepped alone, bit for bit, where a lone problem
takes a step kernel of its own: FP64 at p = 2 with integer columns (608 polyhedra
of long rows), and at most one polyhedron per SM (rows of 4 to 18 blocks,
52 to 125 polyhedra, and 216 beyond the rule)."""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import _lib
from lymph3d_apsc_gb300 import ensemble as E
from test_gpu_batch import _gvals, _prepared

pytestmark = pytest.mark.gpu

BFS = dict(agglomeration="bfs", jitter=0.15, seed=2)
WIDE = dict(n=8, bc="reference", agglomeration="bfs", group=(8, 100), jitter=0.15, seed=1)   # a row of 18 blocks


@pytest.mark.parametrize("precision,specs", [
    (_lib.FP64, [(dict(n=10, group=(4, 12), **BFS), 2, 1e-4), (dict(n=4, group=(4, 12), **BFS), 2, 1e-4)]),
    (_lib.FP64, [(dict(n=5, agglomeration="hex"), p, 1e-4) for p in (1, 2, 3)]),
    (_lib.MIXED, [(dict(n=5, agglomeration="hex"), p, 1e-4) for p in (1, 2, 3)]),
    (_lib.FP64, [(dict(n=5, group=(4, 12), **BFS), p, 1e-4) for p in (1, 2, 3)]),
    (_lib.MIXED, [(dict(n=5, group=(4, 12), **BFS), p, 1e-4) for p in (1, 2, 3)]),
    (_lib.FP64, [(WIDE, p, 1e-4) for p in (1, 2, 3, 4)]),
    (_lib.MIXED, [(WIDE, p, 1e-4) for p in (1, 2, 3)]),
    (_lib.MIXED, [(dict(n=6, agglomeration="hex"), p, 1e-4) for p in (1, 3)]),
    # absorbing sides: the damping products keep one order whatever the CTA's size
    (_lib.FP64, [(dict(n=3, bc="absorbing", **BFS), p, 1e-4) for p in (1, 2, 3, 4)]),
    (_lib.MIXED, [(dict(n=3, bc="absorbing", **BFS), p, 1e-4) for p in (1, 2, 3, 4)]),
    (_lib.MIXED_MF, [(dict(n=3, bc="absorbing", **BFS), p, 1e-4) for p in (1, 2, 3, 4)]),
])
def test_batch_equals_problems_alone(require_gpu, precision, specs):
    batch_solvers = [_prepared(s, precision) for s in specs]
    alone = [_prepared(s, precision) for s in specs]
    b = E.Batch(batch_solvers)
    b.run(_gvals(batch_solvers, 21))
    for s, a in zip(batch_solvers, alone):
        a.run_steps(a.dt, 1e9, max_steps=21)
        assert np.array_equal(s.get_state(_lib.SLOT_UN), a.get_state(_lib.SLOT_UN)), (a.degree, a.n_poly)
    b.close()
    for x in batch_solvers + alone:
        x.close()
