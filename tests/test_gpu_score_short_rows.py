"""The exact scorer at short rows (up to 28 dims, in registers) and with fewer queries than its tiles hold: bit-exact
against the sequential multiply-then-add restatement, and the time of absent queries."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,dim", [(1, 1, 4), (1, 127, 8), (2, 128, 12), (4, 129, 16), (31, 1000, 20), (32, 257, 24),
                                     (32, 300, 28), (33, 300, 28), (33, 300, 16), (65, 129, 4), (5, 400, 36), (17, 200, 44)])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "shifted"])
def test_short_rows_are_bit_exact(torch_cuda, m, n, dim, shift):
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


@pytest.mark.parametrize("dim", [20, 100])
def test_absent_queries_cost_nothing(torch_cuda, dim):
    # six queries of a tile of sixteen: at most what sixteen take (with copies of the last query in the absent ones'
    # places 1.4 and 2.4 times that)
    torch = torch_cuda
    n = 100_000
    q = torch.randn((16, dim), device="cuda")
    v = torch.randn((n, dim), device="cuda")
    out = torch.zeros((16, n), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    us = {}
    for m in (6, 16):
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(50):
                hss.vector_score(q.data_ptr(), v.data_ptr(), out.data_ptr(), m, n, dim, n, stream)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 20)
        us[m] = best
    assert us[6] < 1.25 * us[16], us
