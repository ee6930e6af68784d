"""The batch's step kernels (batch.cu: by grid, tile shape, highest degree and absorbing
faces): with shape 0 every grid gives the problems alone, bit for bit; the other shapes
give one result whatever the grid, equal to the problems alone up to another grouping of
the same sums (FP64 1e-11 relative after 20 steps, the bar of test_gpu_batch.py; FP32
blocks no further from FP64 than three times what the problems alone are).  One problem of
p = 2 has integer columns, with rows of up to 19 blocks."""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import _lib
from lymph3d_apsc_gb300 import ensemble as E
from test_gpu_batch import _gvals, _prepared

pytestmark = pytest.mark.gpu

BFS = dict(agglomeration="bfs", jitter=0.15, seed=1)
INT2 = (dict(n=12, bc="reference", group=(4, 24), **BFS), 2, 1e-4)
SETS = {
    "low": [(dict(n=4, group=(4, 12), **BFS), 1, 1e-4), (dict(n=4, group=(4, 12), **BFS), 2, 1e-4)],
    "low with integer columns": [(dict(n=4, group=(4, 12), **BFS), 1, 1e-4), INT2],
    "all": [(dict(n=3, group=(4, 12), **BFS), p, 1e-4) for p in (1, 2, 3, 4)] + [INT2],
    "absorbing": [(dict(n=3, bc="absorbing", **BFS), p, 1e-4) for p in (1, 2, 3, 4)],
}
STEPS = 20


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("name", list(SETS))
def test_every_kernel_of_the_batch(require_gpu, tmp_path, monkeypatch, name, precision):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("LYMPH_TUNE_CACHE", str(cache))
    solvers = [_prepared(s, precision) for s in SETS[name]]
    b = E.Batch(solvers)
    b.autotune(trial_steps=1, use_cache=False)
    b.close()
    key = cache.read_text().split()[0]
    if name != "low" and name != "absorbing":
        rp, _ = solvers[-1].pattern()
        assert solvers[-1].n_poly >= 608 and np.diff(rp).max() > 16 and np.diff(rp).mean() >= 8
    start = [(s.get_state(_lib.SLOT_U0), s.get_state(_lib.SLOT_UN)) for s in solvers]
    g = _gvals(solvers, STEPS)

    def reset():
        for s, (u0, un) in zip(solvers, start):
            s.set_state(_lib.SLOT_U0, u0)
            s.set_state(_lib.SLOT_UN, un)

    alone = []
    for s in solvers:
        s.run_steps(s.dt, 1e9, max_steps=STEPS)
        alone.append(s.get_state(_lib.SLOT_UN))
    ref = alone
    if precision != _lib.FP64:
        ref = []
        for spec in SETS[name]:
            r = _prepared(spec, _lib.FP64)
            r.run_steps(r.dt, 1e9, max_steps=STEPS)
            ref.append(r.get_state(_lib.SLOT_UN))
            r.close()
    for shape in (0, 1, 2):
        first = None
        for ctas in (1, 3, 4):
            cache.write_text(f"{key} {ctas * 152} 1 {shape}\n")
            b = E.Batch(solvers)
            assert b.schedule() == (ctas * 152, 1, shape)
            reset()
            b.run(g)
            b.close()
            got = [s.get_state(_lib.SLOT_UN) for s in solvers]
            for u, a, r in zip(got, alone, ref):
                if shape == 0:
                    assert np.array_equal(u, a)
                elif precision == _lib.FP64:
                    assert np.linalg.norm(u - a) <= 1e-11 * np.linalg.norm(a)
                else:
                    assert np.linalg.norm(u - r) <= 3.0 * np.linalg.norm(a - r) + 1e-12 * np.linalg.norm(r)
            first = first or got
            assert all(np.array_equal(u, f) for u, f in zip(got, first))
    for s in solvers:
        s.close()
