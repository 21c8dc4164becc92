"""The brick query beyond one pass and without its workspace, bit for bit against the plain query: more than 2^24 points
(offset outputs, a reused workspace, a short last pass whose bricks are sparse where the full pass's are staged), and
the plain kernel in its place when the workspace cannot be allocated."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
LO, HI = (-1.0, -1.1, -0.9), (1.0, 0.9, 1.1)


def _equal(want, a, b):
    for w, x, y in zip(want, a, b):
        assert (y is None) == (not w)
        if w:
            assert torch.equal(x.view(torch.int32), y.view(torch.int32))


@pytest.mark.parametrize("rest", [1, 4099, (1 << 24) + 7])
def test_more_points_than_a_pass(rest):
    from voxneus_b200 import ops

    torch.manual_seed(1)
    grid = torch.randn(1, 1, 64, 64, 64, device=DEV)
    pts = torch.rand((1 << 24) + rest, 3, device=DEV) * 2.2 - 1.1
    a = ops.field_query(grid, LO, HI, pts, sdf=True, grad=True, normal=True)[:3]
    for want in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
        _equal(want, a, ops.field_query_sorted(grid, LO, HI, pts, *map(bool, want))[:3])


def test_no_room_for_the_workspace(monkeypatch):
    from voxneus_b200 import ops

    torch.manual_seed(2)
    grid = torch.randn(1, 1, 40, 40, 40, device=DEV)
    pts = torch.rand(30_001, 3, device=DEV) * 2.0 - 1.0
    a = ops.field_query_sorted(grid, LO, HI, pts, True, True, True)[:3]
    real, tried = torch.empty, []

    def empty(*args, **kw):
        if kw.get("dtype") is torch.uint8:
            tried.append(args)
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*args, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    for want in ((1, 1, 1), (1, 0, 0)):
        _equal(want, a, ops.field_query_sorted(grid, LO, HI, pts, *map(bool, want))[:3])
    assert len(tried) == 2


@pytest.mark.parametrize("res", [(48, 50, 52), (600, 600, 560)], ids=["counted in shared memory", "in device memory"])
@pytest.mark.parametrize("kind", ["outside", "nan", "cell", "five cells", "six cells", "runs"])
def test_crowded_points(res, kind):
    """Points of few cells among 32 neighbours, answered in the order they came: to the line between them and
    bricks from both sides, and crowded stretches beside scattered ones."""
    from voxneus_b200 import ops

    torch.manual_seed(4)
    grid = torch.randn(1, 1, *res, device=DEV)
    n = 40_961
    pts = torch.rand(n, 3, device=DEV) * 2.0 - 1.0
    cell = 2.0 / max(res)
    if kind == "outside":
        pts += 4.0
    elif kind == "nan":
        pts[:] = float("nan")
    elif kind == "cell":
        pts = 0.3 + 0.5 * cell * torch.rand(n, 3, device=DEV)
    elif kind.endswith("cells"):
        at = torch.arange(n, device=DEV) % (5 if kind == "five cells" else 6)
        pts = (torch.rand(6, 3, device=DEV) * 1.6 - 0.8)[at]
    else:
        pts[: n * 9 // 10] = 0.2
    a = ops.field_query(grid, LO, HI, pts, sdf=True, grad=True, normal=True, corners=True)[:3]  # the plain kernel
    for want in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1)):
        _equal(want, a, ops.field_query_sorted(grid, LO, HI, pts, *map(bool, want))[:3])


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("tiny", [1e-30, 1e-33, 1e-36, 1e-40])
def test_vanishing_gradient_along_one_axis(axis, tiny):
    """Differences too small for the division from the reciprocal beside ordinary ones: layers of ~1e-30 and less between
    layers of 1, so that the gradient along the layers is tiny and the one across them is not."""
    from voxneus_b200 import ops

    torch.manual_seed(5)
    grid = torch.randn(1, 1, 45, 47, 52, device=DEV) * tiny
    grid.transpose(2, 2 + axis)[:, :, ::2] = 1.0
    pts = torch.rand(60_000, 3, device=DEV) * 2.0 - 1.0
    a = ops.field_query(grid, LO, HI, pts, sdf=True, grad=True, normal=True)[:3]
    _equal((1, 1, 1), a, ops.field_query_sorted(grid, LO, HI, pts, True, True, True)[:3])
