"""The hash table's adjoint against float64 sums of the same contributions: runs of 4 (points, short batches) and
of 8 (long batches of rays), samples that stay in a cell and that do not, single samples and remainders of a
run, gradients that are zero here and there or everywhere, level counts that fill a block's rows or not,
levels partly open and closed, a wider row stride.

An entry is a float32 sum of c contributions in any order: c - 1 roundings of at most 2^-24 of the sum of
magnitudes each, plus the 6 of a contribution (weights, product). The bound takes c + 6 of them.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
PRIMES = (1, 2654435761, 805459861)


@pytest.mark.parametrize("levels,rays,samples,as_points,active,sparse", [
    (16, 1, 1, True, None, 0.0),
    (16, 3, 3, False, None, 0.0),
    (1, 11, 17, False, None, 0.5),
    (3, 40, 33, True, 2.5, 0.3),
    (32, 50, 21, False, 20.25, 0.0),
    (16, 2049, 128, False, None, 0.6),   # runs of 8
    (16, 4099, 64, False, 10.5, 0.0),    # runs of 8, the last one short
    (16, 300, 64, False, None, 1.0),     # nothing to scatter
])
def test_table_gradient(levels, rays, samples, as_points, active, sparse):
    from voxneus_b200 import ops

    gen = torch.Generator(device=DEV).manual_seed(levels * 1000 + rays)
    log2 = 12
    cfg = ops.HashConfig(n_levels=levels, log2_size=log2)
    p, ld = rays * samples, 2 * levels + 4
    o = torch.rand(rays, 3, device=DEV, generator=gen) * 0.6 - 0.3
    d = torch.nn.functional.normalize(torch.randn(rays, 3, device=DEV, generator=gen), dim=1)
    mid = (torch.rand(rays, samples, device=DEV, generator=gen) * 0.7).sort(1)[0].contiguous()
    lo, hi = (-1.0,) * 3, (1.0,) * 3
    x = ((o[:, None] + d[:, None] * mid[..., None]).reshape(-1, 3) + 1.0) / 2.0
    x = x.clamp(0.0, 1.0).contiguous()
    g = torch.randn(p, ld, device=DEV, generator=gen)
    g = g * (torch.rand(p, 1, device=DEV, generator=gen) >= sparse)
    emb = torch.zeros(levels, 1 << log2, 2, device=DEV)
    if as_points:
        ops.hash_backward(emb, cfg, active, x, None, None, None, 1, None, None, p, g, ld)
    else:
        ops.hash_backward(emb, cfg, active, None, o, d, mid, samples, lo, hi, p, g, ld)
    lw = list(cfg.level_weights(active))
    for l in range(levels):
        s = x * float(cfg.resolutions[l])   # float32, as the kernel's cells and weights
        c = s.floor()
        f = (s - c).double()
        want, mag = (torch.zeros(1 << log2, 2, dtype=torch.float64, device=DEV) for _ in range(2))
        hits = torch.zeros(1 << log2, dtype=torch.float64, device=DEV)
        gl = g[:, 2 * l:2 * l + 2].double() * float(torch.tensor(lw[l], dtype=torch.float32))
        for k in range(8):
            bits = ((k >> 2) & 1, (k >> 1) & 1, k & 1)
            w = torch.ones(p, dtype=torch.float64, device=DEV)
            h = torch.zeros(p, dtype=torch.int64, device=DEV)
            for a in range(3):
                w = w * (f[:, a] if bits[a] else 1.0 - f[:, a])
                h = h ^ ((c[:, a].long() + bits[a]) * PRIMES[a])
            h = h & ((1 << log2) - 1)
            want.index_add_(0, h, w[:, None] * gl)
            mag.index_add_(0, h, (w[:, None] * gl).abs())
            hits.index_add_(0, h, torch.ones_like(w))
        bound = (hits[:, None] + 6.0) * 2.0 ** -24 * mag
        assert bool(((emb[l].double() - want).abs() <= bound).all()), f"level {l}"
