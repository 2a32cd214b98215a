"""The exact scorer's tiles: every tile shape the launcher picks, at the edges of its query and doc tiles,
with a partial last stage of dims, and with matrices that are only 4-byte aligned. Bit-exact against the
sequential multiply-then-add restatement."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,dim", [(1, 1, 4), (2, 129, 36), (3, 37889, 32), (4, 300, 100), (5, 65, 28), (16, 64, 64),
                                     (17, 130, 132), (32, 18944, 128), (33, 19000, 20), (64, 18945, 40)])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "shifted"])
def test_vector_score_tiles_are_bit_exact(torch_cuda, m, n, dim, shift):
    torch = torch_cuda
    rng = np.random.default_rng(m * 1000 + n + dim)
    q = rng.standard_normal((m, dim)).astype(np.float32)
    v = rng.standard_normal((n, dim)).astype(np.float32)
    ld = n + 3
    dq = torch.zeros(m * dim + 4, dtype=torch.float32, device="cuda")
    dv = torch.zeros(n * dim + 4, dtype=torch.float32, device="cuda")
    dq[shift:shift + m * dim] = torch.tensor(q.reshape(-1), device="cuda")
    dv[shift:shift + n * dim] = torch.tensor(v.reshape(-1), device="cuda")
    out = torch.full((m, ld), 7.0, dtype=torch.float32, device="cuda")
    hss.vector_score(dq.data_ptr() + 4 * shift, dv.data_ptr() + 4 * shift, out.data_ptr(), m, n, dim, ld)
    torch.cuda.synchronize()
    s = np.zeros((m, n), np.float32)
    for d in range(dim):
        s = s + np.outer(q[:, d], v[:, d])
    got = out.cpu().numpy()
    assert (got[:, :n].view(np.uint32) == s.view(np.uint32)).all()
    assert (got[:, n:] == 7.0).all()
