"""The training pass's tiles: batches, features and hidden units at the edges of the 32 x 32 tiles, the
8-row output blocks, the 256-unit chunks and the four-way k split, against the float64 restatement."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss
from oracle import mlp_ref

pytestmark = pytest.mark.gpu

# an FP32 sum of n rounded products of random signs errs by about sqrt(n) 2^-24 of its terms' norm; four
# layers of sums of at most 700 terms, against the largest gradient
GRAD_RTOL = 2e-4


@pytest.mark.parametrize("din,h,B", [(5, 32, 1), (32, 33, 31), (33, 64, 33), (64, 31, 128), (397, 256, 512), (130, 257, 65),
                                     (17, 300, 700), (600, 40, 129)])
def test_gradients_at_tile_edges(torch_cuda, din, h, B):
    torch = torch_cuda
    rng = np.random.default_rng(din + h + B)
    m = hss.ThresholdModel(din, h, device=0, seed=3)
    p = m.get_params() + (rng.standard_normal(m.param_count) * 0.01).astype(np.float32)
    m.set_params(p)
    X = rng.standard_normal((B, din)).astype(np.float32)
    t = rng.standard_normal(B).astype(np.float32)
    dX, dT = torch.tensor(X, device="cuda"), torch.tensor(t, device="cuda")
    g, loss = m.gradients(dX.data_ptr(), dT.data_ptr(), B)
    loss_ref, g_ref = mlp_ref.loss_and_grad(p.astype(np.float64), X, t, din, h, 0.0)
    assert abs(loss - loss_ref) <= 1e-4 * max(1.0, loss_ref)
    assert np.abs(g - g_ref).max() <= GRAD_RTOL * np.abs(g_ref).max()
    again, _ = m.gradients(dX.data_ptr(), dT.data_ptr(), B)
    assert (again.view(np.uint32) == g.view(np.uint32)).all()
