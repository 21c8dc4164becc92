"""Lattice queries at the sizes that take bricks: 2^18 points and more in cells with whole stencils, 3 M and more over
the whole grid and beyond; ragged bricks, odd grid rows, an unaligned grid, reversed bounds, the widest spacing. The
positions, the oracle and the bounds are those of the small lattices' test, which the plain kernel answers."""

import pytest
from test_gpu_lattice_brick import test_lattice_matches_point_query as matches_point_query

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,lat,lo,hi,offset", [
    ((64, 64, 64), (64, 64, 64), -0.5, 0.5, 0),
    ((64, 48, 80), (71, 61, 65), -0.4, 0.6, 0),
    ((37, 41, 29), (65, 66, 67), -0.8, 0.8, 0),
    ((64, 64, 64), (64, 65, 66), 0.3, -0.6, 1),
    ((200, 200, 200), (64, 65, 66), -0.53, 0.53, 0),
    ((64, 64, 64), (11, 200, 200), 0.1, 0.6, 0),
    ((48, 50, 52), (150, 151, 140), -1.0, 1.0, 0),
    ((33, 33, 33), (160, 150, 140), -1.05, 1.05, 0),
    ((96, 100, 90), (153, 153, 150), -1.0, 1.0, 1),
])
def test_large_lattices(res, lat, lo, hi, offset):
    matches_point_query(res, lat, lo, hi, offset)
