"""Lattice queries in bricks (spacings below ~1.7 voxels) against the point query of the same positions:
brick edges, lattices smaller than a brick, grid rows of whole 16-byte groups and not, an unaligned grid,
the widest spacing that takes bricks and the next that does not, reversed and partial bounds (points
outside the grid clamp to its border), a lattice finer than the grid.

The SDF keeps the point query's bits. The normal of an interior cell blends the differences before the
division by 2 eps and multiplies by reciprocals: six roundings of 2^-24 more or fewer on a gradient of
length near 1 here, so 1e-5 bounds it with room; border cells keep the bits.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _coords(lo, hi, n):
    """The lattice's coordinates: steps from lo in the first half, back from hi in the second, each product
    and sum rounded to float32 (torch.linspace on the device fuses them)."""
    lo, hi = np.float32(lo), np.float32(hi)
    step, i = np.float32((hi - lo) / np.float32(n - 1)), np.arange(n, dtype=np.float32)
    return torch.from_numpy(np.where(np.arange(n) < n // 2, lo + step * i, hi - step * (np.float32(n - 1) - i))).to(DEV)


@pytest.mark.parametrize("res,lat,lo,hi,offset", [
    ((64, 64, 64), (40, 40, 40), -1.0, 1.0, 0),       # 1.6 voxels a point
    ((64, 48, 80), (41, 33, 65), -1.0, 1.0, 0),       # ragged bricks
    ((37, 41, 29), (30, 35, 24), -1.0, 1.0, 0),       # odd rows: 4-byte copies
    ((64, 64, 64), (40, 40, 40), -1.0, 1.0, 1),       # a grid 4 bytes off 16
    ((96, 96, 96), (55, 56, 57), -1.0, 1.0, 0),       # 1.7 voxels a point: around the limit
    ((64, 64, 64), (20, 20, 20), -1.0, 1.0, 0),       # 3.3 voxels a point: the plain kernel
    ((33, 33, 33), (100, 90, 70), -1.2, 1.1, 0),      # finer than the grid, beyond its border
    ((64, 64, 64), (33, 9, 3), 0.9, -0.4, 0),         # reversed and partial, thinner than a brick
    ((4, 4, 4), (7, 5, 9), -1.0, 1.0, 0),
])
def test_lattice_matches_point_query(res, lat, lo, hi, offset):
    from voxneus_b200 import ops

    torch.manual_seed(sum(res) + sum(lat))
    ax = [torch.linspace(-1.0, 1.0, r, device=DEV) for r in res]
    x, y, z = torch.meshgrid(*ax, indexing="ij")
    f = (x * x + 0.8 * y * y + 1.1 * z * z).sqrt() - 0.4 + 0.1 * x + 0.002 * torch.randn(res, device=DEV)
    store = torch.empty(f.numel() + 4, device=DEV)
    grid = store[offset:offset + f.numel()].view(1, 1, *res)
    grid.copy_(f)
    b = (-1.0,) * 3, (1.0,) * 3
    sdf, nrm = ops.field_query_lattice(grid, *b, lat, (lo,) * 3, (hi,) * 3)
    pts = torch.stack(torch.meshgrid(*[_coords(lo, hi, n) for n in lat], indexing="ij"), -1)
    s, _, n, _, _ = ops.field_query(grid, *b, pts.reshape(-1, 3).contiguous(), sdf=True, normal=True)
    assert torch.equal(sdf, s)
    assert float((nrm - n).abs().max()) <= 1e-5
    only, _ = ops.field_query_lattice(grid, *b, lat, (lo,) * 3, (hi,) * 3, normal=False)
    none, n2 = ops.field_query_lattice(grid, *b, lat, (lo,) * 3, (hi,) * 3, sdf=False)
    assert torch.equal(only, s) and none is None and torch.equal(n2, nrm)
