"""The fused stencil's two ways through a tile, a warp for few vertices and the whole block for many, against a
dense float64 evaluation: grids with fewer tiles than resident blocks (blocks of one tile) and with many,
every vertex active, thinly scattered ones, one crowded region among scattered ones (both ways in one block),
sizes that leave cut tiles on every axis, one tile, no vertex at all. The result repeats bit for bit.

An output sums 7 terms of about 10 roundings each on differences of values up to 4 apart: 1e-5 of the largest
output bounds it with room (70 roundings of 2^-24 are 4e-6).
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("res,scatter,crowd", [
    ((64, 64, 64), 1.0, None),
    ((64, 64, 64), 0.003, None),
    ((5, 6, 33), 1.0, None),
    ((3, 3, 3), 1.0, None),
    ((37, 50, 70), 0.02, (10, 30)),
    ((160, 150, 140), 0.002, (40, 70)),    # 175 tiles a slot of 8 blocks and more: several tiles a block
    ((200, 180, 260), 0.05, (0, 60)),      # more tiles than blocks
    ((64, 64, 64), 0.0, None),
])
def test_tiles_match_dense(res, scatter, crowd):
    from voxneus_b200 import ops

    gen = torch.Generator(device=DEV).manual_seed(sum(res))
    lo, hi = (-1.0,) * 3, (1.0,) * 3
    f = torch.rand(res, device=DEV, generator=gen) * 2.0 - 1.0
    act = torch.rand(res, device=DEV, generator=gen) < scatter
    if crowd:
        a, b = crowd
        act[a:b, a:b, a:b] = True
    bm = ops.new_bitmap(res, DEV)
    if bool(act.any()):
        ops.vr_mark_corners(act.nonzero(), res, bm)
    fb = ops.new_filtered(res, DEV)
    counts = ops.vr_count(bm, f[None, None].contiguous(), res, lo, hi, 0.0, 0.0, filtered=fb)
    nv = int(act.sum())
    out = torch.zeros(res, device=DEV)
    losses = ops.reg_stencil(f[None, None].contiguous(), fb, res, lo, hi, 0.0, 0.0, counts, 0.1, 5e-4, out)
    again = torch.zeros(res, device=DEV)
    losses2 = ops.reg_stencil(f[None, None].contiguous(), fb, res, lo, hi, 0.0, 0.0, counts, 0.1, 5e-4, again)
    assert torch.equal(out, again) and torch.equal(losses, losses2)

    eps = [float(torch.tensor(2.0) / torch.tensor(float(r - 1))) for r in res]
    m = act[1:-1, 1:-1, 1:-1].double()
    d, want = f.double(), torch.zeros(res, dtype=torch.float64, device=DEV)
    mid = [slice(1, r - 1) for r in res]

    def part(t, axis, step):
        s = list(mid)
        s[axis] = slice(1 + step, res[axis] - 1 + step)
        return t[tuple(s)]

    n = [(part(d, a, 1) - part(d, a, -1)) / (2 * eps[a]) for a in range(3)]
    lap = [(part(d, a, 1) + part(d, a, -1) - 2 * d[tuple(mid)]) / eps[a] ** 2 for a in range(3)]
    length = (n[0] ** 2 + n[1] ** 2 + n[2] ** 2).sqrt()
    inv = 2.0 / max(nv, 1)
    for a in range(3):
        e = m * inv * 0.1 * (1.0 - 1.0 / (length + 1e-8)) * n[a] / (2 * eps[a])
        c = m * inv * 5e-4 * lap[a] / eps[a] ** 2
        part(want, a, 1).add_(e + c)
        part(want, a, -1).add_(c - e)
        want[tuple(mid)] -= 2.0 * c
    assert float((out.double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    k = float(m.sum())
    if k > 0:
        eik = float((m * (length - 1.0) ** 2).sum()) / k
        curv = float((m * (lap[0] ** 2 + lap[1] ** 2 + lap[2] ** 2)).sum()) / k
        assert abs(losses[0].item() - eik) <= 1e-5 * eik and abs(losses[1].item() - curv) <= 1e-5 * curv
