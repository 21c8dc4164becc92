"""Which grids the brick query takes (host arithmetic, no GPU): a grid whose bricks its buckets cannot count goes to the
plain kernel, which needs no workspace."""

import pytest

TILE, BUCKETS, SMEM = 4096, 256, 227 * 1024  # records of a block, buckets, shared memory of a block


def _bricks(res):
    return ((res[0] + 15) // 16) * ((res[1] + 15) // 16) * ((res[2] + 15) // 16)


@pytest.mark.parametrize("res", [
    (512, 512, 512), (1290, 1290, 1290), (2, 64, 16777216), (64, 64, 262144), (2, 2, 16777216), (33, 3, 16777216),
    (2, 65, 16000000), (2, 65, 16519104), (2, 32753, 32777), (2, 32752, 32752), (2, 1025, 1047000), (17, 17, 7400000),
    (2, 2, 16777217), (3, 600000000, 1)])
def test_the_counters_of_a_bucket_fit_or_the_grid_is_not_sorted(res):
    from voxneus_b200 import _lib as L

    n = 1 << 21
    got = int(L.query("vx_field_query_sorted_workspace", n, L.i3(res)))
    if min(res) < 2:
        assert got == 0
        return
    bricks, shift = _bricks(res), 0
    while (bricks - 1) >> shift >= BUCKETS:
        shift += 1
    fits = TILE * 18 + (8 << shift) + 4096 <= SMEM  # 4 KB of static shared memory are room enough
    if not fits or max(res) > 1 << 24:
        assert got == 256  # plain kernel
    if got != 256:
        assert fits and got >= 52 * n + 12 * bricks  # and 8 a brick of the work list, at most 8 a point
