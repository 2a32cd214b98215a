"""In-place filter over sparse postings longer than a tile reads whole: bits against numpy, at tile and segment edges,
and the time of a call, which long segments must not multiply by their number of tiles."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu

SEG, N = 524_288, 700_001  # 32 tiles of 256 words a segment, the second one short


def _docs(n):
    """Tags by doc: short and long postings, spread, in rows, at the edges of tiles and segments, none, all."""
    rng = np.random.default_rng(41)
    hit = np.zeros((12, n), bool)
    hit[0] = rng.random(n) < 5e-4
    hit[1] = rng.random(n) < 4e-3
    hit[2] = rng.random(n) < 0.02
    hit[3] = rng.random(n) < 0.03
    hit[4, 100_000:117_000] = True          # units in a row inside a few tiles
    hit[5, 16383::16384] = True             # the last doc of every 256-word tile
    hit[6, ::16384] = True                  # the first
    hit[7, [0, SEG - 1, SEG, n - 1]] = True
    hit[8] = rng.random(n) < 0.3            # dense
    hit[9] = True
    hit[10, SEG:] = rng.random(n - SEG) < 0.02  # nothing in the first segment
    return hit


def _table(torch, hit, seg, packed):
    tags, n = hit.shape
    bits = np.zeros(n, np.uint64)
    for t in range(tags):
        bits |= hit[t].astype(np.uint64) << np.uint64(t)
    vec = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    # (a row whose postings would be denser than a 64th as bitmaps is kept dense, unless packed)
    return hss.DataTable.build_device(vec.data_ptr(), n, 4, bits.reshape(n, 1), tags, device=0, doc_num_per_segment=seg,
                                      sparse_packed=packed)


def _filter(torch, table, exprs, repeat=1):
    nq = len(exprs)
    s = hss.FullRecallSearcher(table, max_batch=nq, decode_in_place=True)
    f = s.compile_filters(exprs)
    words = table.info["segment_num"] * table.info["doc_num_per_segment"] // 64
    out = torch.full((nq, words), -1, dtype=torch.int64, device="cuda")
    passed = torch.zeros(nq, dtype=torch.int32, device="cuda")
    times = []
    for _ in range(repeat):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        assert s.filter_device(f, nq, out.data_ptr(), words, passed.data_ptr(),
                               torch.cuda.current_stream().cuda_stream) == 0
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return out, passed, min(times)


@pytest.mark.parametrize("packed", [False, True], ids=["bitmap", "packed"])
def test_long_postings_match_numpy(torch_cuda, packed):
    hit = _docs(N)
    table = _table(torch_cuda, hit, SEG, packed)
    one = [(str(t), hit[t]) for t in range(11)]
    two = [("2 AND 3", hit[2] & hit[3]), ("0 OR 5 OR 6 OR 7", hit[0] | hit[5] | hit[6] | hit[7]),
           ("NOT 1", ~hit[1]), ("4 AND NOT 2", hit[4] & ~hit[2]), ("8 AND 10", hit[8] & hit[10])]
    every = " OR ".join(str(t) for t in range(8)) + " OR 10"  # many operands: narrow tiles
    two.append((every, np.logical_or.reduce(hit[list(range(8)) + [10]])))
    for group in (one, two[:5], two):  # the batch's largest operand count sets the tiles' width
        out, passed, _ = _filter(torch_cuda, table, [e for e, _ in group])
        got = np.unpackbits(out.cpu().numpy().view(np.uint8), axis=1, bitorder="little")[:, :N].astype(bool)
        for i, (e, want) in enumerate(group):
            assert (got[i] == want).all(), (e, np.nonzero(got[i] != want)[0][:5])
            assert int(passed[i]) == int(want.sum())


def test_long_segments_cost_no_more_than_short_ones(torch_cuda):
    # 4M docs, postings of 20,000 entries and more in one segment of 256 tiles, of 700 and more in 32 segments:
    # the same bits. A tile that read its postings whole took 14 times as long in the one segment.
    n = 4_194_304
    rng = np.random.default_rng(42)
    hit = np.stack([rng.random(n) < p for p in (0.006, 0.008, 0.010, 0.012, 0.014, 0.015)])
    exprs = ["0 AND 1", "2 OR 3 OR 4", "NOT 5 AND 0", "1 OR 4 AND 5", "3", "0 OR 1 OR 2 OR 3 OR 4 OR 5"] * 8
    ms = {}
    for seg in (131_072, n):
        table = _table(torch_cuda, hit, seg, False)
        out, passed, ms[seg] = _filter(torch_cuda, table, exprs, repeat=20)
        if seg == 131_072:
            first = out.clone()
        else:
            assert torch_cuda.equal(out, first)
    assert ms[n] < 4 * ms[131_072], ms
