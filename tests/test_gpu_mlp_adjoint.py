"""The radiance MLP's adjoint from the forward's ReLU mask, at the sizes where its tiles, row forms and
per-block sums change: a single partial tile, one tile a block, several (the folded form keeps four
tiles' SH values in flight), ragged tails, and every row layout (folded and unfolded compact rows, bulk
full rows, strided and unaligned rows).

Against float64 with the mask the forward wrote. A result is a sum of at most 192 products, each within
2^-22 of its float64 value, accumulated in float32 (at most 24 tensor-core additions a tile, then one
rounded addition a tile): 1e-5 of the largest magnitude bounds every output with room.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
TOL = 1e-5


def _weights(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    return g, r, (0.3 * r(64, 51), 0.1 * r(64), 0.3 * r(3, 64), 0.1 * r(3))


def _unpack(mask):
    bits = torch.arange(32, device=DEV)
    return torch.cat([(mask[:, k:k + 1] >> bits) & 1 for k in (0, 1)], dim=1).double()


def _check(x, ws, colors, mask, g, got):
    """x: full float64 rows; got: (d_hash, d_normal, dW0, db0, dW1, db1)."""
    W0, b0, W1, b1 = (w.double() for w in ws)
    z = x @ W0.T + b0
    on = _unpack(mask)
    clear = z.abs() > 1e-5
    assert bool(((z > 0).double() == on)[clear].all())
    h = z * on
    y = torch.sigmoid(h @ W1.T + b1)
    assert float((colors.double() - y).abs().max()) < 1e-5
    y = colors.double()
    d = g.double() * (1 - y) * y
    dz = (d @ W1) * on
    dx = dz @ W0
    ref = (dx[:, :32], dx[:, 48:51], dz.T @ x, dz.sum(0), d.T @ h, d.sum(0))
    for a, b, name in zip(got, ref, ("d_hash", "d_normal", "dW0", "db0", "dW1", "db1")):
        err = float((a.double() - b).abs().max())
        assert err <= TOL * float(b.abs().max()), (name, err, float(b.abs().max()))


@pytest.mark.parametrize("nr,ns", [(1, 128), (149, 128), (800, 128), (40, 256), (33, 96), (1, 1)])
def test_compact_rows(nr, ns):
    from voxneus_b200 import ops

    g, r, ws = _weights(nr)
    p = nr * ns
    rows = torch.randn(p, 36, device=DEV, generator=g)
    rays_d = torch.nn.functional.normalize(r(nr, 3), dim=-1)
    sh = ops.sh4(rays_d).double().repeat_interleave(ns, 0)
    x = torch.cat([rows[:, :32].double(), sh, rows[:, 32:35].double()], 1)
    full = x.float().contiguous()
    mask = torch.empty(p, 2, dtype=torch.int32, device=DEV)
    colors = ops.mlp_forward(full, *ws, mask)
    cot = r(p, 3)
    got = ops.mlp_backward(rows, *ws, cot, colors, rays_d, ns, mask)
    _check(x, ws, colors, mask, cot, got)
    # without the mask: taken from a forward launch on the same rows
    again = ops.mlp_backward(rows, *ws, cot, colors, rays_d, ns)
    clear = ((x @ ws[0].double().T + ws[1].double()).abs() > 1e-5).all(dim=1)
    for a, b in zip(again[:2], got[:2]):
        assert float((a - b)[clear].abs().max()) <= TOL * float(b.abs().max())


@pytest.mark.parametrize("p,ld,offset", [(1, 52, 0), (127, 52, 0), (128, 51, 0), (129, 57, 0), (20000, 51, 0),
                                         (100003, 52, 0), (100003, 52, 1)])
def test_full_rows(p, ld, offset):
    from voxneus_b200 import ops

    g, r, ws = _weights(p + ld)
    store = torch.randn(p * ld + 8, device=DEV, generator=g)
    rows = store[offset:offset + p * ld].view(p, ld)[:, :51]
    mask = torch.empty(p, 2, dtype=torch.int32, device=DEV)
    colors = ops.mlp_forward(rows, *ws, mask)
    cot = r(p, 3)
    got = ops.mlp_backward(rows, *ws, cot, colors, mask=mask)
    _check(rows.double(), ws, colors, mask, cot, got)
    for a, b in zip(ops.mlp_backward(rows, *ws, cot), got):  # mask and colours recomputed: the same bits
        assert torch.equal(a, b)
