"""Active-vertex marking and compaction against torch: grids whose voxels fill their last word and not, fewer
corners than a block and a remainder, corners outside the grid (clamped), blocks that hold more vertices than
one round of the list, capacities below the count (at a round's edge and not), band and relax predicates.
Integers, so equality.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("res,n,cut", [
    ((2, 3, 5), 1, 0),
    ((33, 31, 37), 1025, 7),
    ((64, 64, 64), 70_001, 0),
    ((64, 64, 64), 3_000_000, 2048),   # nearly every voxel: 16 rounds a block
    ((40, 72, 96), 300_000, 4097),
])
def test_marked_vertices_equal_unique(res, n, cut):
    from voxneus_b200 import ops

    gen = torch.Generator(device=DEV).manual_seed(n)
    size = torch.tensor(res, device=DEV)
    c = (torch.rand(n, 3, device=DEV, generator=gen) * (size + 6)).long() - 3
    bm = ops.vr_mark_corners(c, res, ops.new_bitmap(res, DEV))
    k = torch.minimum(c.clamp(min=0), size - 1)
    want = torch.unique((k[:, 0] * res[1] + k[:, 1]) * res[2] + k[:, 2])
    f = torch.rand(res, device=DEV, generator=gen).view(1, 1, *res).contiguous()
    lo, hi = (-1.0,) * 3, (1.0,) * 3
    for relax, band in ((0.0, 0.0), (0.0, 0.4), (0.8, 0.0), (0.8, 0.4)):
        keep = want
        if band > 0:
            keep = keep[f.view(-1)[keep].abs() < band]
        counts = ops.vr_count(bm, f, res, lo, hi, relax, band)
        if relax > 0 and int(counts[1]) > 0:
            ijk = torch.stack([keep // (res[1] * res[2]), keep // res[2] % res[1], keep % res[2]], -1)
            r = (ijk.double() * 2.0 / (size - 1).double() - 1.0).norm(dim=1)
            assert not bool(((r - relax).abs() < 1e-6).any())  # none where rounding decides
            keep = keep[r < relax]
        cap = max(keep.numel() - cut, 0)
        verts, lin = ops.vr_compact(bm, f, res, lo, hi, relax, band, counts, cap)
        assert torch.equal(lin, keep[:cap])
        assert torch.equal((verts[:, 0] * res[1] + verts[:, 1]) * res[2] + verts[:, 2], keep[:cap])
