"""The radiance MLP's adjoint where gradients or inputs are not finite, or their products overflow.

ReLU's adjoint selects: a hidden unit that is inactive for a sample takes nothing from it, whatever the sample's
gradient. Against float64 with the forward's mask: the same entries are finite, and those agree to 1e-5 of the
largest finite magnitude (float32 products and sums of at most 192 terms a sample, 128 samples a tile).
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _close(got, want, name):
    fine = torch.isfinite(want) & (want.abs() < 3.4e38)
    assert torch.equal(torch.isfinite(got), fine), (name, int((torch.isfinite(got) != fine).sum()))
    if bool(fine.any()):
        err = float((got.double() - want)[fine].abs().max())
        assert err <= 1e-5 * float(want[fine].abs().max()), (name, err)


@pytest.mark.parametrize("kind", ["inf", "nan", "inactive", "overflow", "nan row"])
@pytest.mark.parametrize("form,masked", [("folded", True), ("compact", True), ("compact", False), ("full", True),
                                         ("full", False), ("strided", True), ("strided", False)])
def test_nonfinite_samples_reach_only_what_they_activate(form, masked, kind):
    from voxneus_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(11)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    W0, b0, W1, b1 = ws = (0.3 * r(64, 51), -0.2 - 0.1 * r(64).abs(), 0.3 * r(3, 64), 0.1 * r(3))
    compact = form in ("folded", "compact")
    ns = 128 if form == "folded" else 96
    nr = 300 if form == "folded" else 403  # several tiles a block, a ragged tail unless folded
    p = nr * ns
    ld = 36 if compact else (52 if form == "full" else 57)
    rows = r(p, ld)
    at = torch.tensor([3, 140, p // 2, p - 1], device=DEV)
    cot = r(p, 3)
    if kind in ("inf", "nan"):
        cot[at, torch.tensor([0, 1, 1, 0], device=DEV)] = float(kind)
    elif kind == "inactive":
        rows[at] = 0.0  # z = b0 < 0 in all units of the unfolded forms
        cot[at, 2] = float("inf")
    elif kind == "overflow":  # d x above float32's range, d W1 x within it
        W0[:, 0] *= 0.01
        rows[at[:1], 0] = 14.0
        cot[at[:1]] = 1e38
    else:
        rows[at, 5] = float("nan")
    if compact:
        rays_d = torch.nn.functional.normalize(r(nr, 3), dim=-1)
        if kind == "inactive":
            W0[:, 32:48] = 0.0  # SH(d) too
        sh = ops.sh4(rays_d).repeat_interleave(ns, 0)
        full, extra = torch.cat([rows[:, :32], sh, rows[:, 32:35]], 1).contiguous(), (rays_d, ns)
    else:
        rows = rows[:, :51]
        full, extra = rows, (None, 0)
    mask = torch.empty(p, 2, dtype=torch.int32, device=DEV)
    colors = ops.mlp_forward(full, *ws, mask)
    got = ops.mlp_backward(rows, *ws, cot, colors if masked else None, *extra, mask if masked else None)
    bits = torch.arange(32, device=DEV)
    on = torch.cat([(mask[:, k:k + 1] >> bits) & 1 for k in (0, 1)], 1).bool()
    if kind in ("inactive", "nan row"):
        assert not bool(on[at].any())
    x, y = full.double(), colors.double()
    z = x @ W0.double().T + b0.double()
    h = torch.where(on, z, 0.0)
    d = cot.double() * (1 - y) * y
    dz = torch.where(on, d @ W1.double(), 0.0)
    dx = dz @ W0.double()
    want = (dx[:, :32], dx[:, 48:51], dz.T @ x, dz.sum(0), d.T @ h, d.sum(0))
    for a, b, name in zip(got, want, ("d_hash", "d_normal", "dW0", "db0", "dW1", "db1")):
        _close(a, b, name)
    if kind != "nan row":  # some unit stays inactive for all of these samples in at least one kind
        assert bool(torch.isfinite(got[2]).any()) or bool(on[at].any(0).all())
