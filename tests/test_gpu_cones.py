"""The cone passes against the FP64 oracle at the edges of how links are dealt
out (a warp takes up to eight at a time, fewer when there are few) and of the
traversal's lists: one link, just below and above a batch, several cameras a
sample with empty slots, wide cones that put many boxes on the stack at once,
and enough links for several per warp."""
import numpy as np
import pytest

from fieldcheck import field_stats

pytestmark = pytest.mark.gpu


def _scene(n, k, wide):
    from tsr_b200 import scenes
    sc = scenes.sphere_scene(stride=9 if n > 5000 else 24)
    rng = np.random.default_rng(n + 10 * k)
    sc = sc.subset(np.sort(rng.choice(sc.n, size=min(n, sc.n), replace=False)))
    if k > 1:
        extra = rng.integers(0, sc.cams.shape[0], (sc.n, k - 1)).astype(np.uint32)
        extra[rng.random(extra.shape) < 0.3] = 0xFFFFFFFF
        sc.links = np.concatenate([sc.links, extra], 1)
    if wide:   # a few coarse samples over a fine tree
        sc.scale[:: max(1, sc.n // 3)] *= 40.0
    return sc


@pytest.mark.parametrize("n,k,wide", [(1, 1, False), (7, 1, False), (9, 3, False), (33, 1, True), (700, 2, True),
                                      (30000, 1, False)])
def test_field_matches_oracle(n, k, wide):
    from oracle.pyoracle import Oracle
    from tsr_b200 import core
    sc = _scene(n, k, wide)
    o = Oracle(sc).build_tree()
    tree = core.Tree(core.Samples.from_scene(sc))
    o.occupancy()
    f = o.fields()
    g = core.Occupancy(tree, core.Cameras(sc.cams))
    L = tree.counts["leaves"]
    s = field_stats(f, g, L)
    # a kernel value within FP32 rounding of the acceptance threshold moves a
    # whole term: at most one leaf in a thousand, at least two (fieldcheck)
    allowed = max(2, L // 1000)
    for key in ("emptiness_sum", "sampleness_sum", "emptiness_length", "sampleness_length"):
        assert s[key]["outside"] <= allowed, (key, s[key])
    assert s["cone_count_rel"] <= 1e-12
    states = g.getNodeStates()
    assert int((states != f["states"]).sum()) <= allowed
    # the same kernels removed again leave nothing
    ids = np.arange(sc.n)
    g.eraseSamples(ids, core.Cameras(sc.cams))
    for key in ("emptiness_sum", "sampleness_sum"):
        left = np.abs(g.field(key))
        before = np.asarray(f["e_sum" if key[0] == "e" else "s_sum"])
        # sums of n positive terms and of the same terms negated: 2 n roundings of the largest partial sum
        assert left.max() <= 4 * sc.n * k * 2.0 ** -53 * max(1.0, np.abs(before).max()), key
