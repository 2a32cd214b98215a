"""The launches that a batch's rows and largest K decide: the doc sample's passes."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss
import oracle
from hybridsearchsystem_b200 import data

pytestmark = pytest.mark.gpu

BF16, E4M3 = 2, 3
_WORLD = {}


def _world(n):
    if n not in _WORLD:
        mix = data.Mixture(128, 32, (0.3, 0.9), n_clusters=32, seed=31)
        vec, bits, _ = mix.corpus(n, seed=32)
        _WORLD[n] = (mix, vec, bits, hss.DataTable.build(vec, bits, 32, device=0))
    return _WORLD[n]


def _check(sc, ids, cnt, want):
    ws, wi, wc = want
    for i in range(len(wc)):
        c = int(wc[i])
        assert int(cnt[i]) == c
        assert (ids[i][:c] == wi[i][:c]).all()
        assert (sc[i][:c].view(np.uint32) == ws[i][:c].view(np.uint32)).all()


def test_a_sample_that_does_not_grow_is_taken_once(torch_cuda):
    # an eighth of the corpus holds 4,736 groups of 8 docs: half of them serve K = 2300, not K = 2400, whose
    # sample is the smallest one, kept as lists, in one pass as well
    mix, vec, bits, table = _world(300_000)
    launches = {}
    for k in (2300, 2400):
        s = hss.FullRecallSearcher(table, max_batch=16, method=BF16)
        q = mix.queries(16, seed=33)
        exprs = data.make_filters(mix, 16, seed=34)
        for e, v in zip(exprs, q):
            s.add_query(e, v, k)
        sc, ids, cnt = s.batch_search(out_stride=k)
        _check(sc, ids, cnt, oracle.topk(q, exprs, [k] * 16, vec, bits, threads=8))
        t = s.last_times()
        assert t["retries"] == 0
        launches[k] = t["launches"]
    assert launches[2400] == launches[2300]


@pytest.mark.parametrize("method,n,nq,k", [(BF16, 300_000, 256, 8), (E4M3, 100_000, 16, 10)], ids=["bf16", "e4m3"])
def test_a_replayed_batch_is_planned_as_a_direct_one(torch_cuda, method, n, nq, k):
    # a small K: the same sample (its thresholds, bit for bit), the same docs kept and the same launches, whether
    # they are replayed from a graph, which is shared by other K, or not
    torch = torch_cuda
    mix, vec, bits, table = _world(n)
    s = hss.FullRecallSearcher(table, max_batch=nq, method=method)
    q = mix.queries(nq, seed=35)
    exprs = data.make_filters(mix, nq, n_tags=(1, 2), seed=36)
    f = s.compile_filters(exprs)
    d_q = torch.from_numpy(q).to("cuda:0")
    sc = torch.zeros((nq, k), dtype=torch.float32, device="cuda:0")
    ids = torch.zeros((nq, k), dtype=torch.int64, device="cuda:0")
    cnt = torch.zeros(nq, dtype=torch.int32, device="cuda:0")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    seen = []
    for graphs in (False, True, True):  # direct, captured, replayed
        s.set_graphs(graphs)
        assert s.search_device(d_q.data_ptr(), nq, f, [k] * nq, sc.data_ptr(), ids.data_ptr(), cnt.data_ptr(), k,
                               stream.cuda_stream) == 0
        stream.synchronize()
        seen.append((s.last_thresholds(nq)[0].tobytes(), s.last_candidate_counts(nq).tobytes(),
                     s.last_times()["launches"], s.last_times()["retries"]))
    assert s.graph_stats()["replays"] == 1
    assert seen[1:] == [seen[0]] * 2
    _check(sc.cpu().numpy(), ids.cpu().numpy(), cnt.cpu().numpy(), oracle.topk(q, exprs, [k] * nq, vec, bits, threads=8))


@pytest.mark.parametrize("k,spread", [(31, 0), (32, 2), (100, 2)])
def test_the_8_bit_select_step_is_spread_over_the_device(torch_cuda, k, spread):
    # two more launches from K = 32 on (rows of 128 dims); results exact either way
    mix, vec, bits, table = _world(100_000)
    launches = []
    for kk in (1, k):
        s = hss.FullRecallSearcher(table, max_batch=3, method=E4M3)
        q = mix.queries(3, seed=37)
        exprs = ["1", "2 OR 3", "NOT 4"]
        for e, v in zip(exprs, q):
            s.add_query(e, v, kk)
        sc, ids, cnt = s.batch_search(out_stride=kk)
        _check(sc, ids, cnt, oracle.topk(q, exprs, [kk] * 3, vec, bits, threads=8))
        assert s.last_times()["retries"] == 0
        launches.append(s.last_times()["launches"])
    assert launches[1] - launches[0] == spread


def test_the_k_of_one_plan_share_a_graph(torch_cuda):
    # 400,000 docs, 4 queries: K up to 32 are planned with one pass (12.2 K <= 512), K from 33 to 256 with two;
    # every other part of the plan is the same for them
    torch = torch_cuda
    mix, vec, bits, table = _world(400_000)
    s = hss.FullRecallSearcher(table, max_batch=4, method=BF16)
    s.set_graphs(True)
    q = mix.queries(4, seed=38)
    exprs = ["1", "2 OR 3", "NOT 4", "5"]
    f = s.compile_filters(exprs)
    d_q = torch.from_numpy(q).to("cuda:0")
    sc = torch.zeros((4, 256), dtype=torch.float32, device="cuda:0")
    ids = torch.zeros((4, 256), dtype=torch.int64, device="cuda:0")
    cnt = torch.zeros(4, dtype=torch.int32, device="cuda:0")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    captures = []
    for k in (1, 10, 32, 50, 100, 200, 256):
        assert s.search_device(d_q.data_ptr(), 4, f, [k] * 4, sc.data_ptr(), ids.data_ptr(), cnt.data_ptr(), 256,
                               stream.cuda_stream) == 0
        stream.synchronize()
        captures.append(s.graph_stats()["captures"])
        _check(sc.cpu().numpy(), ids.cpu().numpy(), cnt.cpu().numpy(),
               oracle.topk(q, exprs, [k] * 4, vec, bits, threads=8))
    assert captures == [1, 1, 1, 2, 2, 2, 2]
