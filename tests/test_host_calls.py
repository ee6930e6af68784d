"""The library's host side on a fake CUDA runtime (fake_cudart.c): which calls it
makes, and what it does when one fails.  No GPU."""
import re
import struct

import pytest

from lymph3d_apsc_gb300 import mesh as M
from fake_runtime import run

SOLVER = """
m = M.cube(3, bc="reference", agglomeration="bfs", seed=1, group=(4, 12))
s = MatrixFree(m, 3, 1e-4, precision=_lib.{precision})
s.MAKE_MATRICES_FREE()
"""


def _fnv(*parts):
    h = 1469598103934665603
    for p in parts:
        for b in p:
            h = (h ^ b) * 1099511628211 % 2**64
    return h


def test_the_mesh_hash_is_formed_with_the_context(tmp_path):
    """A checkpoint's save and load copy the two states and nothing else; the hash in
    the file is that of the mesh descriptor's arrays."""
    path = tmp_path / "c.ckpt"
    save, load = run(SOLVER.format(precision="FP64") + f"""
fake.fake_clear(); s.save_checkpoint({str(path)!r}, 0.5, 3); out(calls())
fake.fake_clear(); s.load_checkpoint({str(path)!r}); out(calls())
""", tmp_path)
    assert save.count("d") == 2 and save.count("u") == 0
    assert load.count("u") == 2 and load.count("d") == 0
    m = M.cube(3, bc="reference", agglomeration="bfs", seed=1, group=(4, 12))
    parts = [struct.pack("<4i", m.n_node, m.n_tet, m.n_poly, len(m.mat))]
    parts += [a.tobytes() for a in (m.coords, m.tet_vert, m.tet_poly, m.tet_mat, m.neigh, m.fun_tag, m.mat)]
    raw = path.read_bytes()
    assert struct.pack("<Q", _fnv(*parts)) in raw[:128]


@pytest.mark.parametrize("precision", ["FP64", "MIXED", "MIXED_MF"])
@pytest.mark.parametrize("nth", [1, 7, 17, 20])
def test_a_failed_launch_of_a_run_is_reported(tmp_path, precision, nth):
    """The nth launch of 40 steps fails (the 17th: the counter at the end of the graph of 16
    steps; the matrix-free run's first converts the state): an error, not a graph that
    leaves a step out; the next run is whole."""
    failed, log, again, log2 = run(SOLVER.format(precision=precision) + f"""
fake.fake_clear(); fake.fake_fail_launch({nth})
try:
    s.run_steps(s.dt, 1.0, max_steps=40); out(False)
except LymphError:
    out(True)
out(calls()); fake.fake_clear()
s.run_steps(s.dt, 1.0, max_steps=40); out(True); out(calls())
""", tmp_path)
    assert "!" in log and failed
    if "[" in log2:   # else the graph was whole before the failure
        assert log2[log2.index("["):log2.index("]")].count("X") == 16
    assert log2.count("G") == 2 and log2[log2.rindex("G"):].count("X") == 8


@pytest.mark.parametrize("precision", ["FP64", "MIXED", "MIXED_MF"])
@pytest.mark.parametrize("nth", [1, 2, 9, 31])
def test_a_failed_launch_of_a_batch_is_reported(tmp_path, precision, nth):
    failed, log = run(SOLVER.format(precision=precision) + f"""
b = E.Batch([s])
fake.fake_clear(); fake.fake_fail_launch({nth})
try:
    b.run(np.zeros((1, 32))); out(False)
except LymphError:
    out(True)
out(calls())
""", tmp_path)
    assert "!" in log and failed


@pytest.mark.parametrize("timed", [False, True])
def test_the_reported_time_holds_every_kernel_of_a_run(tmp_path, timed):
    """run_steps' first event comes before the first kernel (matrix-free: the conversion
    of the first state), its last after the last."""
    log, = run(SOLVER.format(precision="MIXED_MF") + f"""
fake.fake_clear(); s.run_steps(s.dt, 1.0, max_steps=21, kernel_timing={timed}); out(calls())
""", tmp_path)
    log = "".join(c for c in log if c in "EKXG")
    assert log[0] == "E" and log[-1] == "E" and "K" in log


def test_a_schedule_tuned_on_other_kernels_is_not_taken(tmp_path):
    """Entries under the key of the kernels without integer columns, in the user's cache file
    and in the default one of their time, leave the batch at its default schedule; a key
    tells the blocks that are multiplied in integer columns."""
    home = tmp_path / "home"
    (home / ".cache").mkdir(parents=True)
    blocks, sched, default = run(SOLVER.format(precision="FP64") + f"""
import os
out(int(s.n_blocks))
old = f"sm152_prec0_p3b{{s.n_blocks}} 152 1 2\\n"
open(os.environ["LYMPH_TUNE_CACHE"], "w").write(old)
b = E.Batch([s]); out(b.schedule()); b.close()
del os.environ["LYMPH_TUNE_CACHE"]; os.environ["HOME"] = {str(home)!r}
open({str(home / ".cache" / "lymph3d_gb300_tune2.txt")!r}, "w").write(old)
b = E.Batch([s]); out(b.schedule())
""", tmp_path)
    assert sched == default == [608, 0, 0]
    keys = run("""
import os
for n in (3, 10):
    s = MatrixFree(M.cube(n, agglomeration="bfs", seed=1, group=(4, 12)), 2, 1e-4)
    s.MAKE_MATRICES_FREE()
    b = E.Batch([s]); b.autotune(1, False); b.close()
    out([int(s.n_blocks), open(os.environ["LYMPH_TUNE_CACHE"]).read().split()[-4]])
""", tmp_path)
    for (nb, key), ints in zip(keys, (False, True)):
        assert re.search(rf"_p2b{nb}" + (rf"i{nb}$" if ints else "$"), key), key


@pytest.mark.parametrize("precision", ["FP64", "MIXED_MF"])
def test_the_tuner_times_what_runs(tmp_path, precision):
    """A trial's timed steps are one launch of a graph, as in Batch.run, with no launch of the
    host's between its two events."""
    log, = run(SOLVER.format(precision=precision) + """
b = E.Batch([s]); fake.fake_clear(); b.autotune(3, False); out(calls())
""", tmp_path)
    trials = re.sub(r"\[.*?\]", "", log)                  # without what is captured
    timed = re.findall(r"E([^E]*)E", trials)
    assert len(timed) >= 8 and set(timed) == {"G"}
    assert "K" not in trials and "X" not in trials


@pytest.mark.parametrize("sms,staged,ints", [(152, True, True), (100, False, True), (200, True, False)])
def test_rules_in_ctas_per_sm_ask_the_device(tmp_path, sms, staged, ints):
    """125 polyhedra take the kernel that stages their rows in dynamic shared memory up to one
    polyhedron per SM, 737 of p = 2 the integer columns from four per SM on."""
    got = run("""
import os, re
fake.fake_dynamic_smem.restype = ctypes.c_size_t
s = MatrixFree(M.cube(5, agglomeration="hex"), 2, 1e-4)
s.MAKE_MATRICES_FREE(); fake.fake_dynamic_smem(); s.run_steps(s.dt, 1.0, max_steps=3)
out(fake.fake_dynamic_smem() > 0)
s = MatrixFree(M.cube(10, agglomeration="bfs", seed=1, group=(4, 12)), 2, 1e-4)
s.MAKE_MATRICES_FREE(); b = E.Batch([s]); b.autotune(1, False)
out(re.search(r"i\\d+", open(os.environ["LYMPH_TUNE_CACHE"]).read()) is not None)
""", tmp_path, FAKE_SMS=str(sms))
    assert got == [staged, ints]


@pytest.mark.parametrize("n", [2, 6, 8])
def test_the_mesh_hash_of_every_size(tmp_path, n):
    """48, 1,296 and 3,072 tetrahedra: ids of one and of two bytes, negative neighbours, the
    hash formed in place and by a thread: FNV-1a over the bytes of the arrays."""
    path = tmp_path / "c.ckpt"
    run(f"""
m = M.cube({n}, bc="reference", agglomeration="tet", jitter=0.1)
s = MatrixFree(m, 1, 1e-4); s.MAKE_MATRICES_FREE(); s.save_checkpoint({str(path)!r}, 0.5, 3)
""", tmp_path)
    m = M.cube(n, bc="reference", agglomeration="tet", jitter=0.1)
    parts = [struct.pack("<4i", m.n_node, m.n_tet, m.n_poly, len(m.mat))]
    parts += [a.tobytes() for a in (m.coords, m.tet_vert, m.tet_poly, m.tet_mat, m.neigh, m.fun_tag, m.mat)]
    assert struct.pack("<Q", _fnv(*parts)) in path.read_bytes()[:128]
