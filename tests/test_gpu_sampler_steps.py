"""The multistep sampler against its own module functions, step by step: the depths after k + 1 steps are
those after k steps with up_sample's new ones put in by cat_z_vals. A lane takes a run of
consecutive samples: lengths around each multiple of 32, fewer samples than lanes, the longest ray, one to 32 new samples
a step, random and evenly spaced draws, with and without an occupancy mask.

Both paths form products and sums in double and round them once to float32; their order differs, so a value
near a rounding boundary (about one in 2^28) may differ by an ulp. None is expected in 10^5 values; one
differing ray in 200 is let through.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("n0,per,steps,perturb,occ", [
    (64, 16, 4, True, True),     # 64, 80, 96, 112: the training ray
    (64, 16, 4, False, False),
    (2, 1, 6, True, False),      # the shortest lists
    (31, 1, 3, False, True),     # 31, 32, 33
    (33, 31, 3, True, False),    # 33, 64, 95
    (65, 32, 2, False, True),    # 65, 97
    (96, 1, 2, True, True),      # 96, 97
    (127, 1, 3, False, False),   # 127, 128, 129
    (160, 32, 3, True, True),    # 160, 192, 224: up to 256 samples
    (40, 20, 1, True, False),
])
def test_steps_equal_module_functions(n0, per, steps, perturb, occ):
    from voxneus_b200 import ops

    rays = 200
    gen = torch.Generator(device=DEV).manual_seed(n0 * 1000 + per)
    lo, hi = (-1.0,) * 3, (1.0,) * 3
    ax = torch.linspace(-1.0, 1.0, 48, device=DEV)
    x, y, z = torch.meshgrid(ax, ax, ax, indexing="ij")
    grid = ((x * x + y * y + 1.3 * z * z).sqrt() - 0.5 + 0.02 * torch.randn(48, 48, 48, device=DEV, generator=gen))
    grid = grid.view(1, 1, 48, 48, 48).contiguous()
    o = torch.nn.functional.normalize(torch.randn(rays, 3, device=DEV, generator=gen), dim=1) * 2.5
    d = torch.nn.functional.normalize(0.4 * torch.randn(rays, 3, device=DEV, generator=gen) - o, dim=1)
    t_rand = torch.rand(rays, n0, device=DEV, generator=gen)
    u = torch.rand(steps, rays, per, device=DEV, generator=gen)
    mask = torch.rand(16, 16, 16, device=DEV, generator=gen) < 0.7 if occ else None

    def run(k):
        return ops.sample_multistep(grid, lo, hi, o, d, None, None, n0, per * k, k, perturb,
                                    t_rand if perturb else None, u[:k].contiguous() if perturb and k else None, mask,
                                    lo if occ else None, hi if occ else None)

    before = run(0)[0]
    for k in range(steps):
        pts = o[:, None, :] + d[:, None, :] * before[..., None]
        sdf = ops.field_query(grid, lo, hi, pts.reshape(-1, 3).contiguous())[0].view(rays, -1)
        new = ops.up_sample(o, d, before, sdf, per, 64.0 * 2 ** k, det=not perturb, u=u[k] if perturb else None,
                            occupancy=mask, occ_min=lo, occ_max=hi)
        want, _ = ops.cat_z_vals(before, new)
        got, dists, mid = run(k + 1)
        assert int((got != want).any(1).sum()) <= 1, f"step {k}: {int((got != want).any(1).sum())} rays differ"
        assert torch.equal(dists[:, :-1], got[:, 1:] - got[:, :-1]) and torch.equal(dists[:, -1], dists[:, -2])
        assert torch.equal(mid, got + dists * 0.5)
        before = got
