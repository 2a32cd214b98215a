"""The rank statistics of a doc sample (features): the same whether a query's sample is held in shared memory whole or
walked again for every statistic."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss
from hybridsearchsystem_b200 import data

pytestmark = pytest.mark.gpu

BF16 = 2


def test_statistics_of_long_samples(torch_cuda):
    # a sample of 32,768 docs, all of them past some filters: batches up to as many queries as SMs hold it whole,
    # larger ones 20,480 docs of it (both are passes on SM pairs, so their scores are the same)
    torch = torch_cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mix = data.Mixture(128, 32, (0.3, 0.9), n_clusters=32, seed=61)
    vec, bits, _ = mix.corpus(200_000, seed=62)
    table = hss.DataTable.build(vec, bits, 32, device=0)
    nq = min(sms + 1, 256)
    q = torch.from_numpy(mix.queries(nq, seed=63)).to("cuda:0")
    exprs = ["", "1 OR 2 OR 3", "4", "NOT 5"] * (nq // 4) + [""] * (nq % 4)
    rows = {}
    for n in (nq, nq - 1):
        s = hss.FullRecallSearcher(table, max_batch=n, method=BF16)
        f = s.compile_filters(exprs[:n])
        x = torch.zeros((n, s.feature_dim()), dtype=torch.float32, device="cuda:0")
        torch.cuda.synchronize()
        s.features(q.data_ptr(), n, f, np.resize(np.array([1, 100, 1000, 64], np.uint32), n), x.data_ptr(),
                   torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        rows[n] = x.cpu().numpy()
    assert np.isfinite(rows[nq]).all()
    assert (rows[nq][:nq - 1].view(np.uint32) == rows[nq - 1].view(np.uint32)).all()
