"""Pass A's share of the corpus follows the doc sample that was asked for, a sixteenth of the corpus in the 8-bit form:
every third 256-doc tile for batches on SM pairs, although the sample taken is a little smaller."""
import pytest

import hybridsearchsystem_b200 as hss
from hybridsearchsystem_b200 import data

pytestmark = pytest.mark.gpu

E4M3 = 3


def test_pass_a_is_a_third_of_the_corpus(torch_cuda):
    torch = torch_cuda
    n, nq, k = 2_500_000, 256, 10
    mix = data.Mixture(128, 16, (0.3, 0.9), n_clusters=256, seed=71)
    vec, bits = mix.corpus_device(n)
    torch.cuda.synchronize()
    table = hss.DataTable.build_device(vec.data_ptr(), n, 128, bits, 16, device=0)
    del vec
    s = hss.FullRecallSearcher(table, max_batch=nq, method=E4M3)
    q = torch.from_numpy(mix.queries(nq, seed=72)).to("cuda:0")
    sc = torch.zeros((nq, k), dtype=torch.float32, device="cuda:0")
    ids = torch.zeros((nq, k), dtype=torch.int64, device="cuda:0")
    cnt = torch.zeros(nq, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    assert s.search_device(q.data_ptr(), nq, s.compile_filters([""] * nq), [k] * nq, sc.data_ptr(), ids.data_ptr(),
                           cnt.data_ptr(), k, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert s.last_times()["retries"] == 0
    # a query's list holds pass A's docs first, those of every third tile, then the others
    for i in range(0, nq, 8):
        from_a = s.last_candidates(i)[1] // 256 % 3 == 0
        assert from_a.any() and not from_a.all()
        assert from_a[:from_a.sum()].all(), i
