"""The TOPK operator on lists of up to a few thousand entries, which are sorted whole or cut at a lower bound of the
K-th key first, on both sides of that line: equal to a sort by (score descending, location ascending)."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 512, 513, 1000, 1024, 1025, 4096, 4097])
@pytest.mark.parametrize("levels", [0, 4], ids=["real", "equal scores"])
def test_short_lists(torch_cuda, n, levels):
    torch = torch_cuda
    rng = np.random.default_rng(n + levels)
    sc = (rng.integers(-2, levels - 2, n) * 0.5 if levels else rng.standard_normal(n)).astype(np.float32)
    loc = rng.permutation(1 << 16)[:n].astype(np.int32)
    order = np.lexsort((loc, -sc))
    d_sc, d_loc = torch.tensor(sc, device="cuda"), torch.tensor(loc, device="cuda")
    d_n = torch.tensor([n], dtype=torch.int32, device="cuda")
    for k in (1, 2, 16, 255, 256, 257, 500, 512, 1023, 4096):
        o_sc = torch.full((k + 1,), 9.0, dtype=torch.float32, device="cuda")
        o_loc = torch.full((k + 1,), -9, dtype=torch.int32, device="cuda")
        o_n = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        hss.api.topk(d_sc.data_ptr(), d_loc.data_ptr(), d_n.data_ptr(), k, o_sc.data_ptr(), o_loc.data_ptr(), o_n.data_ptr())
        torch.cuda.synchronize()
        m = min(k, n)
        assert int(o_n[0]) == m
        assert (o_loc[:m].cpu().numpy() == loc[order[:m]]).all() and (o_sc[:m].cpu().numpy() == sc[order[:m]]).all()
        assert float(o_sc[m]) == 9.0 and int(o_loc[m]) == -9
