"""The hash table's adjoint on both sides of its lines between single samples, runs of 4 and runs of 8: 2^17 samples x
levels, 8 samples a ray, 2^18 samples. The sums, the oracle and the bound are those of the adjoint's own test."""

import pytest
from test_gpu_hash_adjoint import test_table_gradient as matches_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels,rays,samples,as_points,active,sparse", [
    (16, 1023, 8, False, None, 0.0),     # 130,944: single samples
    (16, 1025, 8, False, None, 0.3),     # 131,200: runs of 4
    (16, 301, 33, False, 12.5, 0.2),     # runs of 4, a remainder of 1
    (16, 2000, 7, False, None, 0.0),     # too few samples a ray: single samples
    (16, 9000, 1, True, None, 0.1),      # points
    (1, 8191, 32, False, None, 0.5),     # 262,112: runs of 4
    (1, 8193, 32, False, None, 0.5),     # 262,176: runs of 8
])
def test_runs_match_sums(levels, rays, samples, as_points, active, sparse):
    matches_sums(levels, rays, samples, as_points, active, sparse)
