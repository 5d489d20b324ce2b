"""Sorting (token, slot) pairs by expert, one CTA or a cluster: every pair has one row, in its expert's range, and the work list covers them."""
import pytest
import torch

from metrale_inference_alpha_b200.ops.moe_cuda import SortedPairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K", [(3, 2), (511, 8), (512, 8), (2700, 9), (9000, 8)])
@pytest.mark.parametrize("align,tile_rows,lo,E", [(1, 64, 0, 257), (1, 128, 5, 100), (128, 32, 0, 64)])
def test_pairs_sorted_by_expert(T, K, align, tile_rows, lo, E):
    g = torch.Generator().manual_seed(T + E)
    idx = torch.randint(0, lo + E + 3, (T, K), generator=g, dtype=torch.int32)          # some outside the local experts
    idx[:, -1] = lo + E - 1                                                              # one that every token asks for
    idx[1, 0] = -1
    sp = SortedPairs(idx.to("cuda:0"), lo, E, tile_rows, align)
    ids = idx.flatten().long() - lo
    local = (ids >= 0) & (ids < E)
    row = sp.pair_row.cpu().long()
    assert (row[~local] == -1).all()
    count = torch.bincount(ids[local], minlength=E)
    tiles = (count + tile_rows - 1) // tile_rows
    size = tiles * align if align > 1 else count
    start = torch.cumsum(size, 0) - size
    assert sp.expert_off.cpu().tolist() == start.tolist() + [int(size.sum())] and int(sp.total_rows) == int(size.sum())
    at = row[local] - start[ids[local]]
    place = at // align * tile_rows + at % align if align > 1 else at                    # of a pair among its expert's
    assert (place >= 0).all() and (place < count[ids[local]]).all() and (at % align < tile_rows).all()
    assert row[local].unique().numel() == int(local.sum())
    back = sp.row_pair.cpu().long()
    assert torch.equal(back[row[local]], local.nonzero()[:, 0])
    if align > 1:
        assert int((back >= 0).sum()) == int(local.sum())
    n = int(tiles.sum())
    assert sp.tile_expert.cpu()[:n].tolist() == torch.repeat_interleave(torch.arange(E), tiles).tolist() and (sp.tile_expert.cpu()[n:] == -1).all()
    j = torch.cat([torch.arange(int(t)) for t in tiles])
    e = sp.tile_expert.cpu()[:n].long()
    assert torch.equal(sp.tile_row0.cpu()[:n].long(), start[e] + j * (align if align > 1 else tile_rows))
    assert torch.equal(sp.tile_nrows.cpu()[:n].long(), torch.minimum(torch.tensor(tile_rows), count[e] - j * tile_rows))
