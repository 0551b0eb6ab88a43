"""Trees deeper than the paths of the dual cells' enumeration fit one 64-bit
word (12 levels), up to the deepest that the build accepts, against the
oracle: the cells' order depends on both words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INVALID = 0xFFFFFFFF


def _scene(fraction):
    """A few samples of a sphere, half of them drawn together and `fraction` as large."""
    from tsr_b200 import scenes
    sc = scenes.sphere_scene(stride=24, seed=3).subset(np.arange(40) * 7)
    m = sc.n // 2
    r = float(np.median(sc.scale)) / fraction
    sc.scale[:m] = r
    sc.pos[:m] = sc.pos[0] + np.random.default_rng(1).normal(0, 4 * r, (m, 3))
    return sc


def _depth(children):
    level, depth = np.array([0]), 0
    while True:
        inner = level[children[level] != INVALID]
        if inner.size == 0:
            return depth
        level = (children[inner][:, None] + np.arange(8)).ravel()
        depth += 1


@pytest.mark.parametrize("fraction,depth", [(16, 11), (32, 12), (64, 13), (16384, 21), (65536, 23)])
def test_tree_matches_oracle(fraction, depth):
    from oracle.pyoracle import Oracle
    from tsr_b200 import core
    sc = _scene(fraction)
    o = Oracle(sc).build_tree()
    t = core.Tree(core.Samples.from_scene(sc), reorder_samples=False)
    on, tn = o.nodes(), t.getNodes()
    assert _depth(on["children"]) == depth
    np.testing.assert_array_equal(tn.children, on["children"])
    np.testing.assert_array_equal(tn.samples_per_node, on["counts"])
    np.testing.assert_array_equal(t.getPermutation(), o.permutation())
    np.testing.assert_array_equal(t.getDualCells(), o.dual_cells())
