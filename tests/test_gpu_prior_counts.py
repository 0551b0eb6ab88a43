"""The count of nodes that the prior queries classify (visited_priors) against
the walk's definition: the leaves of a children block are answered together; a
flagged inner node at most two levels below them is opened, and its eight
children classified for each of those leaves, unless its box is apart from all
the spheres, or inside all of them and read from the table of sums (which
reaches seven levels down)."""
import numpy as np
import pytest

from test_gpu_priors import _geometry

pytestmark = pytest.mark.gpu

INVALID = 0xFFFFFFFF
RADIUS = 25.0      # the default: the limits below are whole eighths of a leaf, no rounding decides
TABLE_ROWS = 8


def _expected(tree, occ):
    from tsr_b200 import core
    depth, parent, corner, size = _geometry(tree)
    ch = tree.getNodes().children
    n = ch.shape[0]
    flagged = (occ.getNodeStates() & core.NODE_FLAG_SAMPLENESS) > 0
    if not flagged[0]:
        return 0
    inner = np.nonzero((ch != INVALID) & flagged)[0]
    inner = inner[inner > 0]
    inner = inner[np.argsort(depth[inner], kind="stable")]
    r2 = (8.0 * RADIUS) ** 2
    total = 0
    for first in range(1, n, 8):
        leaf = np.nonzero(ch[first:first + 8] == INVALID)[0]
        if leaf.size == 0:
            continue
        d, unit = depth[first], size[first] / 8.0
        bits = (leaf[:, None] >> np.arange(3)) & 1
        low, high = bits.min(0), bits.max(0)
        mid = np.where(low == high, np.where(low == 1, 4.0, -4.0), 0.0)
        ext = np.where(low == high, 0.0, 4.0)
        half = 0.5 * size[inner] / unit
        centre = (corner[inner] + 0.5 * size[inner, None] - (corner[first] + size[first])) / unit
        dist = np.abs(centre - mid)
        near = np.maximum(dist - ext - half[:, None], 0.0)
        far = dist + ext + half[:, None]
        down = d + 3 - depth[inner]
        opens = ((near ** 2).sum(1) <= r2 + 0.25) & (down > 0)
        opens &= ~(((far ** 2).sum(1) < r2 - 0.25) & (down < TABLE_ROWS))
        is_open = np.zeros(n, bool)
        is_open[0] = True
        for level in np.unique(depth[inner]):
            k = np.nonzero(depth[inner] == level)[0]
            is_open[inner[k]] = opens[k] & is_open[parent[inner[k]]]
        total += 8 * int(is_open.sum()) * leaf.size
    return total


@pytest.mark.parametrize("stride,keep", [(24, 1), (24, 40), (40, None)])
def test_visited_priors_counts_classified_nodes(stride, keep):
    from tsr_b200 import core, scenes
    sc = scenes.sphere_scene(stride=stride)
    if keep:
        sc = sc.subset(np.arange(keep) * (sc.n // keep))
    tree = core.Tree(core.Samples.from_scene(sc), reorder_samples=False)
    occ = core.Occupancy(tree, core.Cameras(sc.cams))
    want = _expected(tree, occ)
    assert want > 0 and occ.counts["visited_priors"] == want
