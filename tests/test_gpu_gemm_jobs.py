"""The backward GEMMs (gemm_jobs.cuh) on a graph large enough that an input
gradient's tiles fill the GPU without sharing their K, with node and column
counts that are no multiple of a tile, against the FP64 oracle.  Biases of 5
keep every pre-activation positive, so rounding cannot flip a ReLU; the bar is
the 2e-5 of the small graphs' gradient test (FP32 sums over 4,901 nodes of one
scale: sqrt(4901) eps = 4e-6)."""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import surrogate as S
from oracle import mpnn_ref as R
from parity_util import rel
from test_gpu_surrogate import _random_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,H,O", [(24, 64, 12), (21, 60, 10)])
def test_gradients_on_a_large_graph(require_gpu, F, H, O):
    rng = np.random.default_rng(3)
    N, L, G = 4901, 1, 8
    net = S.MPNN(F, O, H=H, L=L, G=G, seed=3)
    flat = net.init_params(3)
    for k, v in net.unpack(flat).items():
        v[...] = 5.0 if k.startswith("b") else v * 0.2
    net.set_params(flat)
    graph = _random_graph(N, rng, G)
    net.set_graph(graph)
    ref = {k: R.bf16_round(v) if k.startswith("W") else v.astype(np.float64) for k, v in net.unpack(flat).items()}
    g64 = tuple(np.asarray(a, np.float64) if a.dtype.kind == "f" else a for a in graph)
    x = rng.standard_normal((N, F)).astype(np.float32)
    t = rng.standard_normal((N, O)).astype(np.float32)
    _, cache = R.forward(ref, x.astype(np.float64), g64, L, keep=True)
    assert min(cache["z0"].min(), cache[0][1].min(), cache[0][4].min()) > 0.1
    loss = net.loss_grad(x, t)
    loss_ref, g_ref = R.loss_and_grad(ref, x.astype(np.float64), g64, t.astype(np.float64), L)
    assert abs(loss - loss_ref) <= 2e-5 * loss_ref
    gd = net.unpack(net.params_and_grads()[1])
    for k in g_ref:
        assert rel(gd[k], g_ref[k]) <= 2e-5, k
    net.close()
