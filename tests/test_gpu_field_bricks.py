"""The query in bricks (vx_field_query_sorted) against the plain query, bit for bit: grid rows of whole
16-byte groups and not, an unaligned grid, bricks cut by the grid's border, fewer points than a tile, tiles
and chunks with remainders, all points in one brick, more bricks than a block's histogram holds, the longest
axis, points outside the box and points that are not numbers, each combination of outputs, and
means of points a brick around each line between staged bricks and sparse ones.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("res,n,spread,offset", [
    ((64, 48, 80), 4097, 1.0, 0),
    ((37, 41, 29), 50_001, 1.2, 0),           # odd rows, cut bricks, points outside
    ((64, 64, 64), 20_480, 1.0, 1),           # a grid 4 bytes off 16
    ((64, 64, 64), 1, 1.0, 0),
    ((96, 96, 96), 100_003, 0.02, 0),         # clustered: 49 chunks of a few bricks
    ((16, 16, 16), 8192, 1.0, 0),             # one brick
    ((64, 64, 64), 10_240, 1.0, 0),           # 160 points a brick: staged and sparse bricks side by side
    ((64, 64, 64), 16_384, 1.0, 0),           # 256
    ((64, 64, 64), 25_600, 1.0, 0),           # a mean of 400: all staged
    ((17, 33, 16), 8191, 1.0, 0),             # bricks of one cell's width
    ((2, 2, 3), 513, 1.0, 0),
    ((600, 600, 560), 30_011, 1.0, 0),        # 50,540 bricks: counted in device memory
    ((2, 3, 1 << 24), 777, 1.0, 0),           # the longest axis that takes bricks: 2^20 bricks in 256 buckets
])
def test_brick_query_matches_plain(res, n, spread, offset):
    from voxneus_b200 import ops

    torch.manual_seed(n)
    count = res[0] * res[1] * res[2]
    store = torch.randn(count + 4, device=DEV)
    grid = store[offset:offset + count].view(1, 1, *res)
    lo, hi = (-1.0, -1.1, -0.9), (1.0, 0.9, 1.1)
    pts = (torch.rand(n, 3, device=DEV) * 2.0 - 1.0) * spread
    if n > 500:
        pts[7, 0], pts[8, 1], pts[9, 2], pts[10] = float("nan"), float("inf"), -float("inf"), 1e30
        pts[11], pts[12] = torch.tensor(lo, device=DEV), torch.tensor(hi, device=DEV)
    a = ops.field_query(grid, lo, hi, pts, sdf=True, grad=True, normal=True)[:3]
    for want in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 0)):
        b = ops.field_query_sorted(grid, lo, hi, pts, *map(bool, want))[:3]
        for w, x, y in zip(want, a, b):
            assert (y is None) == (not w)
            if w:
                assert torch.equal(x.view(torch.int32), y.view(torch.int32))


@pytest.mark.parametrize("scale,bad", [(1.0, None), (1e-25, None), (0.0, None), (1e30, None), (1.0, float("inf")),
                                       (1.0, float("nan"))])
def test_brick_gradients_divide_as_the_plain_query(scale, bad):
    """The differences' division by 2 eps from its reciprocal, and where that is left for the division:
    vanishing, huge and non-finite values."""
    from voxneus_b200 import ops

    torch.manual_seed(3)
    grid = torch.randn(1, 1, 61, 47, 52, device=DEV) * scale
    if bad is not None:
        grid.view(-1)[::977] = bad
    lo, hi = (-1.0, -0.7, -1.3), (1.1, 0.9, 0.8)
    pts = torch.rand(60_000, 3, device=DEV) * 2.0 - 1.0
    a = ops.field_query(grid, lo, hi, pts, sdf=True, grad=True, normal=True)[:3]
    b = ops.field_query_sorted(grid, lo, hi, pts, True, True, True)[:3]
    for x, y in zip(a, b):
        assert torch.equal(torch.isnan(x), torch.isnan(y))
        assert torch.equal(x.nan_to_num(7.0, 1e38, -1e38), y.nan_to_num(7.0, 1e38, -1e38))
