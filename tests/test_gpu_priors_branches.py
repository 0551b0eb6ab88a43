"""The prior queries' rarer branches against the direct evaluation of their
definition (see test_gpu_priors.py): trees deeper than the FP32 lattice of box
corners, which only files can bring, and cone lengths that are not finite,
which must reach the leaves whose sphere takes them in and no others."""
import numpy as np
import pytest

from tsr_b200 import files

from test_gpu_deep_trees import _scene as _deep_scene
from test_gpu_priors import _geometry

pytestmark = pytest.mark.gpu

INVALID = 0xFFFFFFFF


def _definition(tree, occ, radius, queries):
    """(leaf, its depth, the number of leaves its prior sums, their two sums) per query."""
    from tsr_b200 import core
    depth, parent, corner, size = _geometry(tree)
    leaf_node = tree.getLeaves().node_index
    n2l = tree.getLeaves().node_to_leaf_links
    flagged = (occ.getNodeStates() & core.NODE_FLAG_SAMPLENESS) > 0
    el, sl = occ.field("emptiness_length"), occ.field("sampleness_length")
    far = corner + size[:, None]
    levels = [np.nonzero(depth == d)[0] for d in range(1, depth.max() + 1)]
    for l in queries:
        q = leaf_node[l]
        c = corner[q] + 0.5 * size[q]
        r = size[q] * radius
        t = np.where(c < corner, c - corner, np.where(c > far, c - far, 0.0))
        meets = (t[:, 0] * t[:, 0] + t[:, 1] * t[:, 1]) + t[:, 2] * t[:, 2] <= r * r
        for k in levels:   # a node is reached through boxes that meet
            meets[k] &= meets[parent[k]]
        sel = n2l[meets & (n2l != INVALID) & flagged & (depth <= depth[q] + 3)]
        yield l, depth[q], sel.size, el[sel].sum(), sl[sel].sum()


def _deep_field(fraction, tmp_path, radius, pruner=None):
    """A field over a tree that is too deep for the build, loaded from files the oracle's tree is written to."""
    from oracle.pyoracle import Oracle
    from tsr_b200 import core
    sc = _deep_scene(fraction)
    o = Oracle(sc).build_tree()
    files.write_tree(tmp_path / "deep", o.nodes(), o.leaves(), o.dual_cells())
    perm = o.permutation().astype(np.int64)
    ordered = []
    for a in (sc.pos, sc.nrm, sc.scale, sc.conf, sc.links):
        b = np.empty_like(a)
        b[perm] = a
        ordered.append(b)
    params = core.make_params(prior_radius=radius)
    tree = core.Tree.fromFiles(str(tmp_path / "deep"), core.Samples(*ordered), params=params)
    return tree, core.Occupancy(tree, core.Cameras(sc.cams), params, **({"pruner": pruner} if pruner else {}))


# 24 levels: the first depth the lattice does not hold; 30: leaves below its last cell
@pytest.mark.parametrize("fraction,depth,radius", [(1 << 17, 24, 25.0), (1 << 17, 24, 3.3), (1 << 23, 30, 25.0)])
def test_priors_of_deep_trees_follow_their_definition(fraction, depth, radius, tmp_path):
    tree, occ = _deep_field(fraction, tmp_path, radius)
    leaf_depth = _geometry(tree)[0][tree.getLeaves().node_index]
    assert leaf_depth.max() == depth
    rng = np.random.default_rng(0)
    queries = np.concatenate([rng.choice(np.nonzero(leaf_depth == d)[0], min(12, c), replace=False)
                              for d, c in enumerate(np.bincount(leaf_depth)) if c])
    got = occ.getPriorForEmptiness()
    deep_terms = 0
    for l, d, n, e, s in _definition(tree, occ, radius, queries):
        if n == 0:
            assert np.isnan(got[l]), (l, d)
            continue
        deep_terms += d >= 24
        # the same non-negative FP64 terms in another order: each sum's
        # relative error is at most (terms) 2^-53 on either side
        assert abs(got[l] - e / (e + s)) <= 4 * (n + 64) * 2.0 ** -53, (l, d)
    assert deep_terms > 0


def test_pruned_field_of_a_deep_tree_has_the_plain_signs(tmp_path):
    from tsr_b200 import core
    _, plain = _deep_field(1 << 17, tmp_path, 25.0)
    _, pruned = _deep_field(1 << 17, tmp_path, 25.0, core.Pruner.load())
    np.testing.assert_array_equal(pruned.getOccupancy() > 0, plain.getOccupancy() > 0)


# 3.3: tolerances decide; 5: whole eighths of a leaf; 25: whole, the default
@pytest.mark.parametrize("radius", [3.3, 5.0, 25.0])
def test_infinite_cone_lengths_stay_where_they_belong(radius):
    from tsr_b200 import core, scenes
    sc = scenes.sphere_scene(stride=24)
    sc.conf[sc.n // 2] = np.inf
    params = core.make_params(prior_radius=radius)
    tree = core.Tree(core.Samples.from_scene(sc), params, reorder_samples=False)
    occ = core.Occupancy(tree, core.Cameras(sc.cams), params)
    got = occ.getPriorForEmptiness()
    infinite = ~np.isfinite(occ.field("sampleness_length"))
    assert 0 < infinite.sum() < infinite.size
    rng = np.random.default_rng(1)
    queries = np.unique(np.concatenate([rng.choice(infinite.size, 300), np.nonzero(infinite)[0][:20]]))
    kinds = [0, 0]
    with np.errstate(invalid="ignore"):
        for l, d, n, e, s in _definition(tree, occ, radius, queries):
            want = e / (e + s)
            kinds[int(np.isfinite(e + s))] += 1
            if np.isnan(want):
                assert np.isnan(got[l]), (l, d)
            else:
                assert abs(got[l] - want) <= 4 * (n + 64) * 2.0 ** -53, (l, d)
    assert min(kinds) > 0 or radius == 25.0, kinds
