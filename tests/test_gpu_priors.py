"""The prior queries against a direct evaluation of their definition
(Occupancy.cpp:530-568, SphereNodeStatesChecker.cpp:28-36) from the field's
own cone lengths and node flags: for a leaf, the flagged leaves at most three
levels below it whose box, and every box above it, meets the sphere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INVALID = 0xFFFFFFFF


def _geometry(tree):
    """Depth, parent and FP64 corner of every node, by the build's recurrence."""
    ch, par = tree.getNodes().children, tree.getNodes().parents
    root = tree.getRootScope()
    n = ch.shape[0]
    depth, corner = np.zeros(n, int), np.zeros((n, 3))
    corner[0] = root[:3]
    level = np.array([0])
    while level.size:
        inner = level[ch[level] != INVALID]
        nxt = []
        for c in range(8):
            k = ch[inner] + c
            depth[k] = depth[inner] + 1
            step = root[3] * 0.5 ** depth[k]
            corner[k] = corner[inner] + np.array([c & 1, (c >> 1) & 1, c >> 2]) * step[:, None]
            nxt.append(k)
        level = np.concatenate(nxt) if nxt else np.zeros(0, int)
    return depth, par, corner, root[3] * 0.5 ** depth


def _check(scene, radius):
    from tsr_b200 import core
    params = core.make_params(prior_radius=radius)
    tree = core.Tree(core.Samples.from_scene(scene), params, reorder_samples=False)
    occ = core.Occupancy(tree, core.Cameras(scene.cams), params)
    depth, parent, corner, size = _geometry(tree)
    leaf_node = tree.getLeaves().node_index
    n2l = tree.getLeaves().node_to_leaf_links
    flagged = (occ.getNodeStates() & core.NODE_FLAG_SAMPLENESS) > 0
    is_leaf = n2l != INVALID
    el, sl = occ.field("emptiness_length"), occ.field("sampleness_length")
    got = occ.getPriorForEmptiness()
    order = np.argsort(depth, kind="stable")
    rng = np.random.default_rng(0)
    L = leaf_node.shape[0]
    # some of every depth
    queries = np.unique(np.concatenate([rng.choice(np.nonzero(depth[leaf_node] == d)[0], min(12, c), replace=False)
                                        for d, c in enumerate(np.bincount(depth[leaf_node])) if c]))
    for l in queries:
        q = leaf_node[l]
        c = corner[q] + 0.5 * size[q]
        r = size[q] * radius
        far = corner + size[:, None]
        t = np.where(c < corner, c - corner, np.where(c > far, c - far, 0.0))
        meets = (t[:, 0] * t[:, 0] + t[:, 1] * t[:, 1]) + t[:, 2] * t[:, 2] <= r * r
        for d in range(1, depth.max() + 1):   # a node is reached through boxes that meet
            k = order[depth[order] == d]
            meets[k] &= meets[parent[k]]
        sel = n2l[meets & is_leaf & flagged & (depth <= depth[q] + 3)]
        e, s = el[sel].sum(), sl[sel].sum()
        if sel.size == 0:
            assert np.isnan(got[l]), l
            continue
        # the same non-negative FP64 terms in another order: each sum's
        # relative error is at most (terms) 2^-53 on either side
        assert abs(got[l] - e / (e + s)) <= 4 * (sel.size + 64) * 2.0 ** -53, (l, depth[q])
    assert queries.size > 0 and L == got.shape[0]


def _scene(kind):
    from tsr_b200 import scenes
    if kind == "one":
        return scenes.sphere_scene(stride=24).subset(np.array([7]))
    if kind == "sphere":
        return scenes.sphere_scene(stride=40)
    if kind == "far":   # coordinates 1e7 root sizes from the origin: corners are rounded coarsely
        sc = scenes.sphere_scene(stride=48)
        sc.pos = sc.pos + 2.0e7
        sc.cams = sc.cams + 2.0e7
        return sc
    return scenes.cluttered_scene(seed=3, n_target=3_000)


# 25: the default, whole eighths of a leaf, boxes touch the sphere exactly;
# 3.3: no whole number; 0.4: a sphere inside the leaf; 400: beyond the root
@pytest.mark.parametrize("kind,radius", [("one", 25.0), ("sphere", 25.0), ("sphere", 3.3), ("sphere", 0.4),
                                         ("sphere", 400.0), ("cluttered", 25.0), ("cluttered", 12.5), ("far", 25.0)])
def test_priors_follow_their_definition(kind, radius):
    _check(_scene(kind), radius)
