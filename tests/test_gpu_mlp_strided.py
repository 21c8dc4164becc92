"""The radiance MLP's forward on rows of any stride and alignment against the same rows at 52 floats (bulk copies): the
same products in the same order, so the same bits in colours and ReLU masks; sizes around a tile, a pair of
tiles and several tiles a block, not-a-number in the columns between the rows. And the adjoint without the mask, with
the colours and without, against the one with both."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("ld,offset", [(51, 0), (51, 1), (52, 2), (53, 0), (56, 0), (56, 4), (56, 1), (64, 0), (129, 3)])
@pytest.mark.parametrize("p", [1, 127, 129, 257, 37_889, 120_003])
def test_strided_rows(ld, offset, p):
    from voxneus_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(p + ld)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    ws = (0.3 * r(64, 51), 0.1 * r(64), 0.3 * r(3, 64), 0.1 * r(3))
    store = torch.full((offset + (p - 1) * ld + 51,), float("nan"), device=DEV)  # ends with the last row's last column
    rows = store[offset:].as_strided((p, 51), (ld, 1))
    rows.copy_(r(p, 51))
    full = torch.zeros(p, 52, device=DEV)
    full[:, :51] = rows
    m0, m1 = (torch.empty(p, 2, dtype=torch.int32, device=DEV) for _ in range(2))
    want = ops.mlp_forward(full[:, :51], *ws, m0)
    got = ops.mlp_forward(rows, *ws, m1)
    assert torch.equal(got, want) and torch.equal(m0, m1)
    assert torch.equal(ops.mlp_forward(rows, *ws), want)
    if p > 40_000 and ld % 4:
        return
    cot = r(p, 3)
    b = ops.mlp_backward(rows, *ws, cot, got, mask=m1)
    for other in (ops.mlp_backward(rows, *ws, cot, got), ops.mlp_backward(rows, *ws, cot)):
        for x, y in zip(other, b):
            assert torch.equal(x, y)
