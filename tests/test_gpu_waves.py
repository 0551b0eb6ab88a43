"""Conflict waves of the sampling pass against the sequential oracle where many
sides want the same leaves: lists of dependent sides longer than a warp, one
leaf claimed several times in a wave, and frontiers of more pairs than the
launch has warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters,per,spread", [(1, 3000, 0.02), (6, 700, 0.05), (40, 64, 0.2), (1, 30000, 1.0)])
def test_tree_matches_oracle(clusters, per, spread):
    from oracle.pyoracle import Oracle
    from tsr_b200 import core, scenes
    sc = scenes.sphere_scene(stride=8, seed=4)
    n = clusters * per
    rng = np.random.default_rng(clusters)
    assert n <= sc.n
    at = rng.choice(sc.n, clusters, replace=False).repeat(per)
    radius = float(np.median(sc.scale))
    for name in ("nrm", "conf", "links"):
        setattr(sc, name, getattr(sc, name)[at])
    sc.pos = sc.pos[at] + rng.normal(0, spread * (radius if clusters > 1 else 40 * radius), (n, 3))
    sc.scale = sc.scale[at] * rng.choice([0.5, 1.0, 2.0], n)
    o = Oracle(sc).build_tree()
    t = core.Tree(core.Samples.from_scene(sc), reorder_samples=False)
    on, tn = o.nodes(), t.getNodes()
    np.testing.assert_array_equal(tn.children, on["children"])
    np.testing.assert_array_equal(tn.samples_per_node, on["counts"])
    np.testing.assert_array_equal(t.getPermutation(), o.permutation())
    np.testing.assert_array_equal(t.getDualCells(), o.dual_cells())
