"""A corpus in the order of its clusters and tags: the doc sample's threshold must be as good as in a random
order, as a sample of single docs would give it. Ids and scores equal the oracle's bit for bit.

The sample is a quarter of the corpus, so it holds about 512 docs of a tag (of 2,047 in a row) and of a
query's cluster (about 2,046 in a row), five times K = 100. A threshold near their K-th best keeps about 4 K
docs; the bounds below leave room for each form's error band (the 8-bit form's band holds most of a cluster)
and are passed by a threshold from fewer than K groups, which keeps every doc of the tag, and by one that
falls to other clusters' scores.
"""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss
import oracle
from hybridsearchsystem_b200 import data

pytestmark = pytest.mark.gpu

N, CLUSTERS, TAGS, K = 130_900, 64, 64, 100  # 1,023 tiles of 128 docs: an odd number, the last one short
SIMT, TF32, BF16, E4M3 = 0, 1, 2, 3


@pytest.fixture(scope="module")
def world(torch_cuda):
    mix = data.Mixture(128, TAGS, (1e-3, 0.5), n_clusters=CLUSTERS, seed=21)
    vec, _, cid = mix.corpus(N, seed=22)
    vec = np.ascontiguousarray(vec[np.argsort(cid, kind="stable")])
    tag = np.arange(N) * TAGS // N
    bits = (np.uint64(1) << tag.astype(np.uint64)).reshape(N, 1)
    return mix, vec, bits, hss.DataTable.build(vec, bits, TAGS, device=0)


@pytest.mark.parametrize("nq", [1, 130])
@pytest.mark.parametrize("method", [SIMT, TF32, BF16, E4M3], ids=["simt", "tf32", "bf16", "e4m3"])
def test_threshold_in_an_ordered_corpus(world, method, nq):
    mix, vec, bits, table = world
    s = hss.FullRecallSearcher(table, max_batch=nq, method=method)
    q = mix.queries(nq, seed=23)
    rng = np.random.default_rng(24)
    tags = [str(int(rng.integers(TAGS))) for _ in range(nq)]
    for exprs, most in ((tags, 2047 if method == E4M3 else 1024), ([""] * nq, 4096)):
        for e, v in zip(exprs, q):
            s.add_query(e, v, K)
        sc, ids, cnt = s.batch_search(out_stride=K)
        ws, wi, wc = oracle.topk(q, exprs, [K] * nq, vec, bits, threads=8)
        for i in range(nq):
            c = int(wc[i])
            assert int(cnt[i]) == c
            assert (ids[i][:c] == wi[i][:c]).all()
            assert (sc[i][:c].view(np.uint32) == ws[i][:c].view(np.uint32)).all()
        kept = s.last_candidate_counts(nq)
        assert s.last_times()["retries"] == 0
        assert kept.mean() <= most, (kept.mean(), kept.max())
