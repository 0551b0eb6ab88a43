"""The order-exact sampling nodes against the oracle where the FP32 filter of
the search is weakest: coordinates far from the origin (corners rounded
coarsely), very small and very large scenes, many samples in one place with
scales that differ, so that searches are long."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    from tsr_b200 import scenes
    sc = scenes.sphere_scene(stride=24, seed=3)
    rng = np.random.default_rng(5)
    if kind.startswith("offset"):
        off = float(kind.split(":")[1])
        sc.pos, sc.cams = sc.pos + off, sc.cams + off
    elif kind.startswith("scale"):
        f = float(kind.split(":")[1])
        sc.pos, sc.scale, sc.cams = sc.pos * f, sc.scale * f, sc.cams * f
    elif kind == "dense":
        sc.pos[: sc.n // 2] = sc.pos[0] + rng.normal(0, 1e-3, (sc.n // 2, 3))
        sc.scale = sc.scale * rng.choice([0.25, 1.0, 16.0], sc.n)
    return sc


@pytest.mark.parametrize("kind", ["offset:1e5", "offset:2e7", "scale:1e-6", "scale:1e7", "dense"])
def test_tree_matches_oracle(kind):
    from oracle.pyoracle import Oracle
    from tsr_b200 import core
    sc = _scene(kind)
    o = Oracle(sc).build_tree()
    t = core.Tree(core.Samples.from_scene(sc), reorder_samples=False)
    on, tn = o.nodes(), t.getNodes()
    np.testing.assert_array_equal(tn.children, on["children"])
    np.testing.assert_array_equal(tn.samples_per_node, on["counts"])
    np.testing.assert_array_equal(t.getPermutation(), o.permutation())
    np.testing.assert_array_equal(t.getDualCells(), o.dual_cells())
