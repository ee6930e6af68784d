"""The forward GEMMs' column tiles (32 to 256 wide by the number of row tiles,
the last one ragged) against the FP64 oracle, at the 2e-5 of the forward test
(FP32 sums of at most 600 terms of one scale: sqrt(600) eps = 1.5e-6 a layer)."""
import numpy as np
import pytest

from lymph3d_apsc_gb300 import surrogate as S
from oracle import mpnn_ref as R
from parity_util import rel
from test_gpu_surrogate import _random_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,O", [(1, 16, 1), (127, 48, 40), (130, 80, 24), (300, 272, 33), (2976, 256, 24), (4900, 96, 24),
                                   (9800, 96, 24)])
def test_forward_matches_oracle(require_gpu, N, H, O):
    rng = np.random.default_rng(N)
    F, L, G = 24, 2, 8
    net = S.MPNN(F, O, H=H, L=L, G=G, seed=3)
    flat = net.init_params(3)
    net.set_params(flat)
    if N > 1:
        graph = _random_graph(N, rng, G)
    else:
        graph = (np.zeros(2, np.int32), np.zeros(0, np.int32), np.zeros(0, np.float32),
                 rng.standard_normal((1, G)).astype(np.float32))
    net.set_graph(graph)
    ref = {k: R.bf16_round(v) if k.startswith("W") else v.astype(np.float64) for k, v in net.unpack(flat).items()}
    g64 = tuple(np.asarray(a, np.float64) if a.dtype.kind == "f" else a for a in graph)
    x = rng.standard_normal((N, F)).astype(np.float32)
    assert rel(net.forward(x), R.forward(ref, x.astype(np.float64), g64, L)) <= 2e-5
    net.close()
