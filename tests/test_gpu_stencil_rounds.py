"""The fused stencil's rounds of eight tiles, where the most crowded are left to the whole block and the rest go to a
warp each: active sets of every density, so that rounds leave none, some and all of their tiles to the block,
and crowded regions among empty ones. Against the dense evaluation and bound of the tiles' own test."""

import pytest
from test_gpu_stencil_tiles import test_tiles_match_dense as matches_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,scatter,crowd", [
    ((128, 120, 130), 0.1, None),
    ((128, 120, 130), 0.3, None),
    ((128, 120, 130), 0.7, None),
    ((128, 120, 130), 1.0, None),
    ((160, 150, 140), 0.1, (64, 68)),
    ((160, 150, 140), 0.0, (30, 90)),
    ((36, 40, 34), 0.3, (8, 20)),
])
def test_rounds_match_dense(res, scatter, crowd):
    matches_dense(res, scatter, crowd)
