"""The cross-shard merge of few entries (a thread each, nothing cut) on both sides of its bound: equal to a stable sort by
(score descending, shard ascending, position ascending)."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shards,k,stride", [(1, 1, 1), (2, 10, 10), (2, 255, 255), (2, 256, 256), (8, 63, 63), (8, 64, 64),
                                             (9, 15, 15), (16, 15, 20), (16, 16, 16), (17, 8, 8), (64, 3, 3), (64, 4, 4),
                                             (4, 100, 30), (4, 30, 100)])
@pytest.mark.parametrize("levels", [0, 3], ids=["real", "equal scores"])
def test_merge_of_few_entries(torch_cuda, shards, k, stride, levels):
    torch = torch_cuda
    rng = np.random.default_rng(shards * 1000 + k + levels)
    nq = 6
    sc, ids, cnt = [], [], []
    for _ in range(shards):
        v = rng.integers(0, levels, (nq, stride)) * 0.5 if levels else rng.standard_normal((nq, stride))
        sc.append(-np.sort(-v.astype(np.float32), axis=1))
        ids.append(rng.integers(0, 1 << 40, (nq, stride)))
        c = rng.integers(0, stride + 1, nq)
        c[0], c[1] = stride, 0
        cnt.append(c.astype(np.int32))
    d_sc, d_id, d_n = ([torch.tensor(x, device="cuda") for x in xs] for xs in (sc, ids, cnt))
    o_sc = torch.full((nq, k + 1), 7.0, dtype=torch.float32, device="cuda")
    o_id = torch.full((nq, k + 1), -7, dtype=torch.int64, device="cuda")
    o_n = torch.full((nq,), -1, dtype=torch.int32, device="cuda")
    hss.merge_shards([x.data_ptr() for x in d_sc], [x.data_ptr() for x in d_id], [x.data_ptr() for x in d_n], nq, stride, k,
                     o_sc.data_ptr(), o_id.data_ptr(), o_n.data_ptr(), k + 1)
    torch.cuda.synchronize()
    got_sc, got_id, got_n = o_sc.cpu().numpy(), o_id.cpu().numpy(), o_n.cpu().numpy()
    for q in range(nq):
        n = [min(int(cnt[s][q]), stride, k) for s in range(shards)]
        allsc = np.concatenate([sc[s][q, :n[s]] for s in range(shards)])
        allid = np.concatenate([ids[s][q, :n[s]] for s in range(shards)])
        order = np.argsort(-allsc, kind="stable")[:k]
        assert got_n[q] == order.size
        assert (got_id[q, :order.size] == allid[order]).all()
        assert (got_sc[q, :order.size] == allsc[order]).all()
        assert (got_id[q, order.size:] == -7).all() and (got_sc[q, order.size:] == 7.0).all()
