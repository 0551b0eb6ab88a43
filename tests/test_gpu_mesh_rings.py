"""Hole filling with few and with many border edges: the ring search keeps its
arrays in shared memory up to 9000 border edges and in global memory above."""
import numpy as np
import pytest

from oracle import pyoracle

from test_mesh_oracle import uv_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv,gone,above", [(12, 10, 0.05, False), (150, 120, 0.02, False), (240, 200, 0.05, True)])
def test_rings_match_oracle(nu, nv, gone, above):
    from tsr_b200 import core
    rng = np.random.default_rng(nu)
    V, T = uv_sphere(nu=nu, nv=nv)
    T = T[rng.random(T.shape[0]) > gone]
    m = core.DualMarchingCells.fromArrays(V, T, min_isle_size=10)
    c, p, _, _, t = pyoracle.mesh_postprocess(V, T, scales=np.zeros(V.shape[0]), min_isle_size=10)
    assert (c["border_edges"] > 9000) == above
    for k in ("border_edges", "holes", "hole_vertices", "hole_triangles", "skipped_rings"):
        assert m.post_counts[k] == c[k], k
    np.testing.assert_array_equal(m.triangles, t)
    np.testing.assert_array_equal(m.positions, p)
