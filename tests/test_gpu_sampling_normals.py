"""Sampling nodes against the oracle for normals that are not of unit length:
the side of a plane that a point lies on does not depend on the length, and
where FP32 cannot hold the products (lengths near 1e-38 and below) the exact
tests have to decide."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [0.5, 1e-11, 1e-13, 1e-38, 1e-40, 1e-42, 1e-100])
def test_tree_matches_oracle(length):
    from oracle.pyoracle import Oracle
    from tsr_b200 import core, scenes
    sc = scenes.sphere_scene(stride=24, seed=3)
    sc.nrm = sc.nrm * length
    o = Oracle(sc).build_tree()
    t = core.Tree(core.Samples.from_scene(sc), reorder_samples=False)
    on, tn = o.nodes(), t.getNodes()
    np.testing.assert_array_equal(tn.children, on["children"])
    np.testing.assert_array_equal(tn.samples_per_node, on["counts"])
    np.testing.assert_array_equal(t.getPermutation(), o.permutation())
    np.testing.assert_array_equal(t.getDualCells(), o.dual_cells())
