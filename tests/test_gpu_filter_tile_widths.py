"""In-place filter at the line between one tile a segment (eight words a thread) and several (four at most), with few and
many operands, for every posting layout: bits against numpy."""
import numpy as np
import pytest

import hybridsearchsystem_b200 as hss

pytestmark = pytest.mark.gpu

TAGS = 12


@pytest.mark.parametrize("seg", [131_072, 131_072 + 128, 262_144 - 128])
@pytest.mark.parametrize("layout", [{}, dict(sparse_packed=True), dict(matrix_posting=True)], ids=["bitmap", "packed", "matrix"])
def test_tile_widths_match_numpy(torch_cuda, seg, layout):
    torch = torch_cuda
    n = 2 * seg - 77  # the second segment short
    rng = np.random.default_rng(51)
    hit = np.stack([rng.random(n) < p for p in np.geomspace(1e-4, 0.6, TAGS)])
    hit[3, seg - 1] = hit[3, seg] = hit[3, n - 1] = True
    bits = np.zeros(n, np.uint64)
    for t in range(TAGS):
        bits |= hit[t].astype(np.uint64) << np.uint64(t)
    vec = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    table = hss.DataTable.build_device(vec.data_ptr(), n, 4, bits.reshape(n, 1), TAGS, device=0, doc_num_per_segment=seg,
                                       **layout)
    words = table.info["segment_num"] * seg // 64
    few = [(str(t), hit[t]) for t in range(TAGS)] + [("3 AND 11", hit[3] & hit[11]), ("0 OR NOT 10", hit[0] | ~hit[10])]
    many = few + [(" OR ".join(map(str, range(11))) + " AND 11", np.logical_or.reduce(hit[:10]) | (hit[10] & hit[11]))]
    for group in (few, many):
        s = hss.FullRecallSearcher(table, max_batch=len(group), decode_in_place=True)
        f = s.compile_filters([e for e, _ in group])
        out = torch.full((len(group), words), -1, dtype=torch.int64, device="cuda")
        passed = torch.zeros(len(group), dtype=torch.int32, device="cuda")
        assert s.filter_device(f, len(group), out.data_ptr(), words, passed.data_ptr(),
                               torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        # a segment's words follow one another; docs past the last are clear
        got = np.unpackbits(out.cpu().numpy().view(np.uint8), axis=1, bitorder="little")
        assert not got[:, n:].any()
        for i, (e, want) in enumerate(group):
            assert (got[i, :n].astype(bool) == want).all(), e
            assert int(passed[i]) == int(want.sum())
