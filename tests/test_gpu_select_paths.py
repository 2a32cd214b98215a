"""The selection kernels' paths against the oracle, ids and scores bit for bit: K on both sides of half the
sample's groups (group maxima, lists of docs), lists rescored whole, cut in one wave and in two, cached and
walked, few and many queries (one CTA per SM or two), dims that are no multiple of 16, filters that leave
fewer docs than K."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss
import oracle
from hybridsearchsystem_b200 import data

pytestmark = pytest.mark.gpu

_WORLD = {}


def _world(n, dim):
    if (n, dim) not in _WORLD:
        mix = data.Mixture(dim, 48, (2e-4, 0.6), n_clusters=40, seed=9)
        vec, bits, _ = mix.corpus(n, seed=10)
        vec[n // 3] = vec[n // 2] = vec[n - 1]  # equal scores
        _WORLD[(n, dim)] = (mix, vec, bits, hss.DataTable.build(vec, bits, 48, device=0, doc_num_per_segment=16384))
    return _WORLD[(n, dim)]


def _check(n, dim, method, nq, topks, sample_docs=32768, cap=1 << 18):
    mix, vec, bits, table = _world(n, dim)
    q = mix.queries(nq, seed=nq + 11)
    exprs = data.make_filters(mix, nq, n_tags=(1, 5), seed=nq + 12)
    exprs[0] = ""
    exprs[-1] = "NOT 5"
    topks = np.resize(np.asarray(topks, np.uint32), nq)
    s = hss.FullRecallSearcher(table, max_batch=nq, method=method, sample_docs=sample_docs, candidate_cap=cap)
    for a, e, k in zip(q, exprs, topks):
        s.add_query(e, a, int(k))
    scores, ids, counts = s.batch_search(out_stride=int(topks.max()))
    want_s, want_i, want_c = oracle.topk(q, exprs, topks.astype(np.int32), vec, bits, threads=8)
    for i in range(nq):
        c = int(want_c[i])
        assert int(counts[i]) == c, (i, exprs[i])
        assert (ids[i, :c] == want_i[i, :c]).all(), (i, exprs[i])
        assert (scores[i, :c].view(np.uint32) == want_s[i, :c].view(np.uint32)).all()


@pytest.mark.parametrize("method", [0, 1, 2, 3], ids=["simt", "tf32", "bf16", "e4m3"])
@pytest.mark.parametrize("nq,k", [(1, 1), (5, 100), (9, 2048), (9, 2049), (150, 513), (3, 4096)])
def test_select_paths_match_the_oracle(torch_cuda, method, nq, k):
    _check(60001, 128, method, nq, [k])


@pytest.mark.parametrize("method,dim", [(0, 100), (0, 36), (1, 32), (1, 352), (2, 64), (2, 704)])
def test_select_paths_at_other_dims(torch_cuda, method, dim):
    _check(20003, dim, method, 40, [1, 10, 300, 1000])


@pytest.mark.parametrize("method", [0, 2, 3], ids=["simt", "bf16", "e4m3"])
@pytest.mark.parametrize("sample_docs,cap", [(512, 1 << 18), (4096, 8192), (60001, 1 << 18)])
def test_small_samples_and_lists(torch_cuda, method, sample_docs, cap):
    _check(60001, 128, method, 17, [3, 128, 256, 257, 1024], sample_docs=sample_docs, cap=cap)


@pytest.mark.parametrize("method", [0, 2], ids=["simt", "bf16"])
@pytest.mark.parametrize("nq", [60, 200], ids=["one_cta", "two_ctas"])
def test_lists_shorter_than_k_keep_every_entry(torch_cuda, method, nq):
    # more than 512 candidates but fewer than K: no K-th best is sought, so the kernel goes from reading
    # the list's length straight to clearing the counter that held it; every warp must have read it first
    n, k = 60001, 3000
    mix, vec, bits, table = _world(n, 128)
    q = mix.queries(nq, seed=71)
    exprs = data.make_filters(mix, nq, n_tags=(1, 2), seed=72, selectivity_range=(0.01, 0.045))
    want_s, want_i, want_c = oracle.topk(q, exprs, np.full(nq, k, np.int32), vec, bits, threads=8)
    assert ((want_c > 512) & (want_c < k)).sum() >= nq // 2
    s = hss.FullRecallSearcher(table, max_batch=nq, method=method)
    for _ in range(20):
        for a, e in zip(q, exprs):
            s.add_query(e, a, k)
        scores, ids, counts = s.batch_search(out_stride=k)
        assert (np.asarray(counts) == want_c).all()
        for i in range(nq):
            c = int(want_c[i])
            assert (ids[i, :c] == want_i[i, :c]).all(), i
            assert (scores[i, :c].view(np.uint32) == want_s[i, :c].view(np.uint32)).all(), i


@pytest.mark.parametrize("method,dim,nq,topks", [
    (3, 384, 1, [1]), (3, 384, 40, [1, 10, 300, 1000]), (3, 256, 130, [2048, 7]), (3, 128, 9, [256, 1024]),
    (2, 704, 7, [745]), (2, 704, 64, [2049, 1, 745]), (1, 352, 5, [1490, 4096])])
@pytest.mark.parametrize("n", [300, 20003])
def test_rescoring_spread_over_the_device(torch_cuda, method, dim, nq, topks, n):
    # (300 docs: every list is rescored whole; a filter that passes fewer docs than K, or none)
    _check(n, dim, method, nq, topks)


@pytest.mark.parametrize("method,dim", [(2, 64), (2, 128), (0, 36), (3, 128)])
@pytest.mark.parametrize("n", [127, 128, 129, 257, 511, 513])
def test_short_lists_around_the_whole_and_wave_limits(torch_cuda, method, dim, n):
    # a corpus no larger than the doc sample: list lengths on both sides of the limits, K around half of them
    _check(n, dim, method, 12, [1, 7, 63, 64, 65, 128, 255])


@pytest.mark.parametrize("sample_docs", [4096, 16384, 60001])
def test_listed_samples_of_short_and_long_segments(torch_cuda, sample_docs):
    # K past half the sample's groups keeps the sample as lists of docs: segments on both sides of the
    # 64 entries at which they are walked one after the other
    _check(60001, 128, 2, 20, [sample_docs // 16 + 1 if sample_docs < 60001 else 4000, 2048], sample_docs=sample_docs)
