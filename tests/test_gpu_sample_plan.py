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
