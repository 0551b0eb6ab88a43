"""Vertex scales of depth maps whose pixels lie at the map's edges: maps one
block wide or high, and every pattern of missing pixels around one pixel."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _check(depths):
    from tsr_b200 import core
    h, w = depths.shape
    m = np.array([[0.01, 0, 0], [0, 0.01, 0], [-0.005 * w, -0.005 * h, 1.0]])
    g = core.DepthImage(depths).triangulate(m, m, np.zeros(3))
    o = pyoracle.depth_triangulate(depths, m, m, np.zeros(3))
    np.testing.assert_array_equal(g.triangles, o["triangles"])
    np.testing.assert_array_equal(g.pixel_to_vertex, o["pixel_to_vertex"])
    np.testing.assert_array_equal(g.scales, o["scales"])   # the same sums in the same order


@pytest.mark.parametrize("h,w", [(2, 2), (2, 33), (33, 2), (3, 3), (17, 257)])
def test_narrow_maps(h, w):
    rng = np.random.default_rng(h * 1000 + w)
    d = 2.0 + 0.01 * rng.standard_normal((h, w))
    _check(d)
    d[rng.random(d.shape) < 0.2] = -1.0
    _check(d)


def test_every_neighbourhood():
    # 3 x 3 patterns of missing pixels, side by side
    rng = np.random.default_rng(1)
    d = 2.0 + 0.005 * rng.standard_normal((16 * 4, 32 * 4))
    for k in range(512):
        y, x = 4 * (k // 32), 4 * (k % 32)
        bits = np.array([(k >> b) & 1 for b in range(9)]).reshape(3, 3)
        d[y:y + 3, x:x + 3][bits == 1] = 0.0
        d[y + 3, x:x + 4] = d[y:y + 4, x + 3] = -1.0
    _check(d)
