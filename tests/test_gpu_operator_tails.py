"""The TOPK operator's cluster path and the Aggregator's launch forms at the sizes where they change:
the one-CTA bound, the sampled bound, lists that need every digit of the key, entries listed more than
once, infinities and NaN; blocks of 4,096 docs, the bounds of one and
two launches. All results exact."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu


def _topk(torch, scores, locs, k):
    d_sc, d_loc = torch.tensor(scores, device="cuda"), torch.tensor(locs.view(np.int32), device="cuda")
    d_n = torch.tensor([len(scores)], dtype=torch.int32, device="cuda")
    o_sc = torch.full((k + 1,), 7.0, dtype=torch.float32, device="cuda")
    o_loc = torch.full((k + 1,), 7, dtype=torch.int32, device="cuda")
    o_n = torch.zeros(1, dtype=torch.int32, device="cuda")
    hss.topk(d_sc.data_ptr(), d_loc.data_ptr(), d_n.data_ptr(), k, o_sc.data_ptr(), o_loc.data_ptr(), o_n.data_ptr())
    torch.cuda.synchronize()
    assert o_sc[k].item() == 7.0 and o_loc[k].item() == 7
    return o_sc.cpu().numpy(), o_loc.cpu().numpy().view(np.uint32), int(o_n.item())


@pytest.mark.parametrize("n,k", [(4096, 1), (4096, 4096), (4097, 4096), (4097, 1), (16384 * 4 + 3, 500), (131072, 100),
                                 (131073, 100), (131073, 4096), (1000003, 1000)])
@pytest.mark.parametrize("form", ["normal", "levels", "equal", "ascending", "extreme"])
def test_topk_operator_at_its_bounds(torch_cuda, n, k, form):
    rng = np.random.default_rng(n * 7 + k)
    scores = {"normal": rng.standard_normal(n) * 0.088, "levels": rng.integers(0, 5, n) * 0.25, "equal": np.full(n, -0.5),
              "ascending": np.arange(n) * 1e-6 - 0.3,
              "extreme": rng.choice([np.inf, -np.inf, 0.0, -0.0, 3e38, -3e38, 1e-42], n)}[form].astype(np.float32)
    locs = rng.permutation(n).astype(np.uint32)
    sc, loc, c = _topk(torch_cuda, scores, locs, k)
    assert c == min(n, k)
    order = np.lexsort((locs, -(scores + 0.0)))[:k]  # -0.0 counts as 0.0
    assert (loc[:c] == locs[order]).all()
    assert (sc[:c] == scores[order]).all()


def test_topk_operator_with_repeated_entries_and_nan(torch_cuda):
    rng = np.random.default_rng(5)
    # 9,000 copies of one entry around rank 60, more than the sort buffer holds
    scores = np.concatenate([np.full(9000, 0.5), rng.uniform(0.6, 0.9, 59), rng.uniform(-1, 0.4, 20000)]).astype(np.float32)
    locs = np.concatenate([np.full(9000, 3), np.arange(10, 69), np.arange(100, 20100)]).astype(np.uint32)
    sc, loc, c = _topk(torch_cuda, scores, locs, 100)
    best = np.sort(scores[9000:9059])[::-1]
    assert c == 100 and (sc[:59] == best).all() and (sc[59:100] == 0.5).all() and (loc[59:100] == 3).all()
    # a positive NaN orders above +inf, by its bits, as before
    scores = (rng.standard_normal(30000) * 0.1).astype(np.float32)
    scores[17] = np.nan
    scores[21] = np.inf
    sc, loc, c = _topk(torch_cuda, scores, np.arange(30000, dtype=np.uint32), 10)
    assert np.isnan(sc[0]) and loc[0] == 17 and loc[1] == 21 and c == 10


@pytest.mark.parametrize("n", [63, 64, 4095, 4096, 4097, 65537, 1 << 20, (1 << 20) + 1, 3000001])
@pytest.mark.parametrize("keep", [0.0, 0.03, 1.0])
def test_aggregator_blocks_compact_in_order(torch_cuda, n, keep):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    words = (n + 63) // 64
    hit = rng.random(words * 64) < keep
    hit[n:] = True  # bits past the last doc are not counted
    bits = np.packbits(hit, bitorder="little").view(np.int64)
    scores = rng.standard_normal(n).astype(np.float32)
    d_bits, d_sc = torch.tensor(bits, device="cuda"), torch.tensor(scores, device="cuda")
    wsb = hss.aggregator_workspace_size(n)
    for noalloc in (False, True):
        o_sc = torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda")
        o_loc = torch.full((n + 1,), 7, dtype=torch.int32, device="cuda")
        cnt = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        ws = torch.zeros(wsb, dtype=torch.uint8, device="cuda")
        if noalloc:
            hss.aggregator_noalloc(d_bits.data_ptr(), d_sc.data_ptr(), None, o_sc.data_ptr(), o_loc.data_ptr(),
                                   cnt.data_ptr(), n)
        else:
            hss.aggregator(d_bits.data_ptr(), d_sc.data_ptr(), None, o_sc.data_ptr(), o_loc.data_ptr(), cnt.data_ptr(), n,
                           ws.data_ptr(), wsb)
        torch.cuda.synchronize()
        at = np.nonzero(hit[:n])[0]
        c = int(cnt.item())
        assert c == at.size
        assert (o_loc.cpu().numpy()[:c] == at).all() and (o_sc.cpu().numpy()[:c] == scores[at]).all()
        assert (o_loc[c:] == 7).all().item()


def test_aggregator_past_the_two_launch_bound(torch_cuda):
    torch = torch_cuda
    n = 16384 * 4096 + 130
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    words = (n + 63) // 64
    hit = torch.rand(words * 64, generator=g, device="cuda") < 0.01
    hit[n:] = False
    bits = (hit.view(words, 64).to(torch.int64) << torch.arange(64, device="cuda")).sum(dim=1)
    scores = torch.randn(n, generator=g, device="cuda")
    o_sc, o_loc = torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    wsb = hss.aggregator_workspace_size(n)
    ws = torch.zeros(wsb, dtype=torch.uint8, device="cuda")
    hss.aggregator(bits.data_ptr(), scores.data_ptr(), None, o_sc.data_ptr(), o_loc.data_ptr(), cnt.data_ptr(), n,
                   ws.data_ptr(), wsb)
    at = torch.nonzero(hit[:n]).view(-1)
    assert int(cnt.item()) == at.numel()
    assert torch.equal(o_loc[:at.numel()].long(), at) and torch.equal(o_sc[:at.numel()], scores[at])
