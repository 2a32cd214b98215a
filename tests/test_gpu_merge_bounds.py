"""The cross-shard merge at its bounds: lists that are empty, short or full, more winners from one shard
than from the others, equal scores across shards, prefixes past the shared-memory buffer, the most shards.
Results equal a stable sort by (score descending, shard ascending, position ascending)."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shards,k,stride,form", [
    (1, 10, 10, "full"), (2, 1, 4, "full"), (8, 1000, 1000, "full"), (8, 1000, 1000, "short"), (8, 1000, 1200, "one"),
    (33, 100, 100, "short"), (64, 4096, 4096, "equal"), (64, 37, 64, "levels"), (7, 50, 20, "full"), (3, 100, 100, "empty"),
    (16, 2000, 2000, "infinite"), (5, 0, 10, "full")])
def test_merge_equals_a_stable_sort(torch_cuda, shards, k, stride, form):
    torch = torch_cuda
    rng = np.random.default_rng(shards * 100 + k)
    nq, out_stride = 5, max(k, 1) + 3
    sc, ids, cnt = [], [], []
    for s in range(shards):
        v = rng.standard_normal((nq, stride)) * 0.1 + (0.5 if form == "one" and s == 2 else 0.0)
        if form == "equal":
            v[:] = 0.25
        elif form == "levels":
            v = rng.integers(0, 4, (nq, stride)) * 0.5
        elif form == "infinite":
            v = rng.choice([np.inf, -np.inf, 0.0, -0.0, 1.0], (nq, stride))
        sc.append(-np.sort(-v.astype(np.float32), axis=1))
        ids.append(rng.integers(0, 1 << 40, (nq, stride)))
        c = np.full(nq, stride)
        if form == "short":
            c = rng.integers(0, stride + 1, nq) * (rng.random(nq) < 0.6)
            c[0] = stride if s == 1 else 1
        elif form == "empty":
            c[:] = 0
        cnt.append(c.astype(np.int32))
    d = lambda xs: [torch.tensor(x, device="cuda") for x in xs]
    d_sc, d_id, d_n = d(sc), d(ids), d(cnt)
    o_sc = torch.full((nq, out_stride), 7.0, dtype=torch.float32, device="cuda")
    o_id = torch.full((nq, out_stride), -7, dtype=torch.int64, device="cuda")
    o_n = torch.full((nq,), -1, dtype=torch.int32, device="cuda")
    hss.merge_shards([x.data_ptr() for x in d_sc], [x.data_ptr() for x in d_id], [x.data_ptr() for x in d_n], nq, stride, k,
                     o_sc.data_ptr(), o_id.data_ptr(), o_n.data_ptr(), out_stride)
    torch.cuda.synchronize()
    got_sc, got_id, got_n = o_sc.cpu().numpy(), o_id.cpu().numpy(), o_n.cpu().numpy()
    for q in range(nq):
        n = [min(int(cnt[s][q]), stride, k) for s in range(shards)]
        allsc = np.concatenate([sc[s][q, :n[s]] for s in range(shards)])
        allid = np.concatenate([ids[s][q, :n[s]] for s in range(shards)])
        order = np.argsort(-(allsc + 0.0), kind="stable")[:k]
        assert got_n[q] == order.size
        assert (got_id[q, :order.size] == allid[order]).all()
        assert (got_sc[q, :order.size] == allsc[order]).all()
        assert (got_id[q, order.size:] == -7).all() and (got_sc[q, order.size:] == 7.0).all()
