"""Waits that run out in the middle of a block's tiles, in every row form of the MLP kernels.

A worker that gives up a wait keeps the issuing warp from issuing more MMAs and copies, so that no barrier has
two phases outstanding when the block drains and leaves. With limits of a few polls the give-ups fall on
any of the waits of the several tiles a block takes; after them the context stays usable and the default
limit gives the bits of before.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("polls", [0, 1, 2, 5])
@pytest.mark.parametrize("form", ["folded", "compact", "full", "strided"])
def test_short_limits_leave_the_context_usable(form, polls):
    from voxneus_b200 import _lib, ops

    g = torch.Generator(device=DEV).manual_seed(7)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    ws = (0.3 * r(64, 51), 0.1 * r(64), 0.3 * r(3, 64), 0.1 * r(3))
    ns = 128 if form == "folded" else 96
    nr = 148 * 5 if form == "folded" else 148 * 7 + 3
    p = nr * ns
    rays_d = torch.nn.functional.normalize(r(nr, 3), dim=-1) if form in ("folded", "compact") else None
    ld = {"folded": 36, "compact": 36, "full": 52, "strided": 57}[form]
    rows = r(p, ld) if rays_d is not None else r(p, ld)[:, :51]
    full = torch.cat([rows[:, :32], ops.sh4(rays_d).repeat_interleave(ns, 0), rows[:, 32:35]], 1).contiguous() \
        if rays_d is not None else rows
    cot = r(p, 3)
    extra = (rays_d, ns) if rays_d is not None else (None, 0)

    def both():
        mask = torch.zeros(p, 2, dtype=torch.int32, device=DEV)
        colors = ops.mlp_forward(full, *ws, mask)
        kept = ops.mlp_backward(rows, *ws, cot, colors, *extra, mask)
        made = ops.mlp_backward(rows, *ws, cot, None, *extra)  # mask and colours from one more forward launch
        return (colors, mask, *kept, *made)

    good = both()
    _lib.query("vx_tensor_core_timeouts")
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    with ops.tc_guard(status, polls):
        both()
    torch.cuda.synchronize()
    n = int(status.item())
    assert n > 0 or polls > 0
    assert _lib.query("vx_tensor_core_timeouts") == n
    again = both()
    torch.cuda.synchronize()
    assert _lib.query("vx_tensor_core_timeouts") == 0
    for a, b in zip(again, good):
        assert torch.equal(a, b)
