"""Compaction of thinly scattered vertices: blocks (32,768 voxels) without any, with a few that go straight to the lists,
and around the line to the lists in shared memory. Integers, so equality, as in the vertex lists' own test."""

import pytest
from test_gpu_vertex_list import test_marked_vertices_equal_unique as marked_equal_unique

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,n,cut", [
    ((96, 96, 96), 5, 0),
    ((96, 96, 96), 400, 3),
    ((96, 100, 96), 1850, 0),      # ~60 a block
    ((96, 100, 96), 2200, 61),     # ~70 a block
])
def test_scattered_vertices(res, n, cut):
    marked_equal_unique(res, n, cut)
