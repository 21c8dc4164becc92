"""The appearance-row kernel: every part alone against the oracle and in one row with the others, for level counts
that leave threads of a row without levels, rows that fill a block, leave a remainder or are fewer, row
strides wider than the columns (the rest untouched), parts in other orders and laid over one another
(the last of hash, SH, normal, pad stays).

Hash features are sums of 8 products of magnitudes up to 1: 16 roundings of 2^-24 bound the difference from the
oracle's order by 1e-6; the other parts are copies or rounded op by op as the oracle's.
"""

import pytest
import torch

from oracle import reference_path as O

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("levels,p", [(1, 1), (2, 63), (3, 64), (5, 65), (16, 1000), (31, 130), (32, 4097)])
def test_rows_of_parts(levels, p):
    from voxneus_b200 import ops
    from voxneus_b200._lib import call, ptr, stream_ptr

    gen = torch.Generator(device=DEV).manual_seed(levels)
    cfg = ops.HashConfig(n_levels=levels, log2_size=10)
    table = torch.rand(levels, 1 << 10, 2, device=DEV, generator=gen) * 2.0 - 1.0
    pts = torch.rand(p, 3, device=DEV, generator=gen) * 1.1 - 0.05
    dirs = torch.nn.functional.normalize(torch.randn(p, 3, device=DEV, generator=gen), dim=1)
    nrm = torch.randn(p, 3, device=DEV, generator=gen)
    nh = 2 * levels

    def rows(ld, sh=-1, normal=-1, pad=-1, hash_=True, active=None):
        out = torch.full((p, ld), 7.5, device=DEV)
        call("vx_appearance_forward", ptr(table) if hash_ else None, levels if hash_ else 0, 10, 2,
             cfg._res_c if hash_ else None, cfg.level_weights(active) if hash_ else None, ptr(pts), None, None, None, 1,
             None, None, p, ptr(out), ld, sh, ptr(dirs), 3, normal, ptr(nrm), pad, stream_ptr(DEV))
        return out

    for active in (None, 0.4 * levels + 0.3):
        ref = O.hash_encode(pts.cpu(), table.cpu(), cfg.resolutions, active)
        assert float((rows(nh, active=active).cpu() - ref).abs().max()) <= 1e-6
    h, s = rows(nh), rows(16, sh=0, hash_=False)
    assert torch.equal(s.cpu(), O.sh4(dirs.cpu()))
    a = rows(nh + 24, sh=nh, normal=nh + 16, pad=nh + 19)
    assert torch.equal(a, torch.cat([h, s, nrm, torch.zeros(p, 1, device=DEV), torch.full((p, 4), 7.5, device=DEV)], 1))
    b = rows(nh + 25, sh=nh + 5, normal=nh + 1)  # normal before SH, gaps
    gap = torch.full((p, 1), 7.5, device=DEV)
    assert torch.equal(b, torch.cat([h, gap, nrm, gap, s, gap.expand(p, 4)], 1))
    c = rows(max(nh, 18), sh=1, normal=3, pad=4)  # over one another
    want = torch.full((p, max(nh, 18)), 7.5, device=DEV)
    want[:, :nh] = h
    want[:, 1:17] = s
    want[:, 3:6] = nrm
    want[:, 4] = 0.0
    assert torch.equal(c, want)


@pytest.mark.parametrize("p,offset,grads", [(1, 0, (True, True)), (127, 0, (True, False)), (129, 1, (False, True)),
                                            (1000, 3, (True, True))])
def test_radiance_parts_equal_rows(p, offset, grads):
    """The module's separate inputs (contiguous, off 16 bytes, expanded) against the MLP on the same rows: the
    same kernels, so the same bits; a part that takes no gradient gets none."""
    from voxneus_b200 import ops
    from voxneus_b200.models import RadianceMLP

    gen = torch.Generator(device=DEV).manual_seed(p)
    mlp = RadianceMLP().to(DEV)
    ws = [mlp.net[0].weight, mlp.net[0].bias, mlp.net[2].weight, mlp.net[2].bias]
    h = torch.randn(p * 32 + 4, device=DEV, generator=gen)[offset:offset + p * 32].view(p, 1, 32)
    v = torch.randn(1, 1, 16, device=DEV, generator=gen).expand(p, 1, 16)
    n = torch.randn(p, 1, 3, device=DEV, generator=gen)
    h, n = h.detach().requires_grad_(grads[0]), n.requires_grad_(grads[1])
    rows = torch.zeros(p, 52, device=DEV)
    rows[:, :51] = torch.cat([h, v, n], -1).detach().view(p, 51)
    x = rows[:, :51].requires_grad_(True)
    cot = torch.randn(p, 3, device=DEV, generator=gen)
    ref = ops.RadianceMLPFn.apply(x, *ws)
    want = torch.autograd.grad((ref * cot).sum(), [x, *ws])
    out = mlp(h, v, n)
    assert out.shape == (p, 1, 3) and torch.equal(out.view(p, 3), ref)
    (out.view(p, 3) * cot).sum().backward()
    assert (h.grad is not None) == grads[0] and (n.grad is not None) == grads[1]
    if grads[0]:
        assert torch.equal(h.grad.view(p, 32), want[0][:, :32])
    if grads[1]:
        assert torch.equal(n.grad.view(p, 3), want[0][:, 48:51])
    for w, g in zip(ws, want[1:]):
        assert torch.equal(w.grad, g)


@pytest.mark.parametrize("change", [lambda t: t.mul_(0.5), lambda t: t.clamp_(0.4, 0.6), lambda t: t.data.mul_(0.5)],
                         ids=["mul_", "clamp_", "data"])
@pytest.mark.parametrize("rows", [False, True])
def test_colours_may_be_changed_in_place_before_the_backward(rows, change):
    """Neither MLP function keeps the tensor it returns, so a caller may change it; the gradients are those of
    the same change out of place (the change's own part is left to autograd: none for .data)."""
    from voxneus_b200 import ops
    from voxneus_b200.models import RadianceMLP

    gen = torch.Generator(device=DEV).manual_seed(5)
    mlp = RadianceMLP().to(DEV)
    ws = [mlp.net[0].weight, mlp.net[0].bias, mlp.net[2].weight, mlp.net[2].bias]
    x = torch.randn(300, 51, device=DEV, generator=gen).requires_grad_(True)
    cot = torch.randn(300, 3, device=DEV, generator=gen)

    def colours():
        return ops.RadianceMLPFn.apply(x, *ws) if rows else mlp(x[:, :32], x[:, 32:48].detach(), x[:, 48:])

    out = colours()
    y = out.detach().clone()
    change(out)
    got = torch.autograd.grad((out * cot).sum(), [x, *ws])
    u = y.clone().requires_grad_(True)
    v = u * 1.0
    change(v)
    (d,) = torch.autograd.grad((v * cot).sum(), u)
    want = torch.autograd.grad(colours(), [x, *ws], d)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
