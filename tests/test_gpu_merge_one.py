"""The cross-shard merge of one shard: its lists as they are, up to their counts and the top K."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,stride", [(1, 1), (0, 4), (512, 512), (513, 600), (2000, 2000), (4096, 4096), (100, 30), (30, 100)])
def test_one_shard(torch_cuda, k, stride):
    torch = torch_cuda
    rng = np.random.default_rng(k + stride)
    nq, out_stride = 5, max(k, 1) + 2
    sc = -np.sort(-rng.standard_normal((nq, stride)).astype(np.float32), axis=1)
    ids = rng.integers(0, 1 << 40, (nq, stride))
    cnt = rng.integers(0, stride + 1, nq).astype(np.int32)
    cnt[0], cnt[1], cnt[2] = stride, 0, stride + 7
    d_sc, d_id, d_n = (torch.tensor(x, device="cuda") for x in (sc, ids, cnt))
    o_sc = torch.full((nq, out_stride), 7.0, dtype=torch.float32, device="cuda")
    o_id = torch.full((nq, out_stride), -7, dtype=torch.int64, device="cuda")
    o_n = torch.full((nq,), -1, dtype=torch.int32, device="cuda")
    hss.merge_shards([d_sc.data_ptr()], [d_id.data_ptr()], [d_n.data_ptr()], nq, stride, k, o_sc.data_ptr(),
                     o_id.data_ptr(), o_n.data_ptr(), out_stride)
    torch.cuda.synchronize()
    for q in range(nq):
        n = min(int(cnt[q]), stride, k)
        assert int(o_n[q]) == n
        assert (o_sc[q, :n].cpu().numpy() == sc[q, :n]).all() and (o_id[q, :n].cpu().numpy() == ids[q, :n]).all()
        assert (o_sc[q, n:] == 7.0).all() and (o_id[q, n:] == -7).all()
