"""The work that a user has this library do, as timed cases.

Each case is one whole call path through the public entry points: the Python
classes of ``tsr_b200.core`` (host arrays in, host arrays out), or the C ABI
of ``include/tsr_core.h`` as ``bench.py`` drives it (samples in pinned host
buffers or in device memory, results read into pinned host buffers that the
program keeps, sized for its largest surface).  Inputs are the seeded scenes of ``tsr_b200.scenes`` with the
shapes and value distributions of the benchmark's workloads.

Paths (``path``):

* ``crust``  -- samples and cameras to the surface: tree, occupancy field, dual
  marching cells.  ``api``: "python" (core.Samples ... extractCrust, with the
  crust's post-processing), "host" (C ABI from pinned buffers, with the
  reordered samples read back, as the reference reorders them in place),
  "device" (C ABI on device-resident samples).
* ``pruned`` -- a kept tree's field with the learned pruner, and its surface.
* ``update`` -- a kept tree and field: 1 % of the samples removed, the surface,
  the same samples added again, the surface.
* ``depth``  -- one depth map to a mesh of samples.
* ``post``   -- isle deletion, hole filling and normals of a surface.
* ``train``  -- the pruner's gradients of one batch.
* ``infer``  -- the pruner's logits of a field's leaves.
"""
import ctypes
import math

import numpy as np
import torch

from tsr_b200 import core, pruner, scenes

# --------------------------------------------------------------------- cases


def listed():
    return [
        # a first look at a capture, or one object of a few thousand samples:
        # launches and host round trips decide
        dict(name="crust_4k", path="crust", api="python", scene="sphere", n=4_000, k=1),
        # the benchmark's unit sphere at full size, with the crust's post-processing
        dict(name="crust_sphere_250k", path="crust", api="python", scene="sphere", n=250_000, k=1),
        # a cluttered capture (outliers, confidences in [0.2, 1]) whose samples
        # were seen by up to three cameras, an odd count
        dict(name="crust_clutter_300k_k3", path="crust", api="device", scene="cluttered", n=300_007, k=3),
        # a medium capture handed over from the caller's host buffers
        dict(name="crust_csg_1m_host", path="crust", api="host", scene="csg", n=1_000_000, k=1),
        # the benchmark's CSG scene, samples already on the device
        dict(name="crust_csg_4m", path="crust", api="device", scene="csg", n=4_000_000, k=1),
        # the benchmark's default workload
        dict(name="crust_heldout_16m", path="crust", api="device", scene="heldout", n=16_000_000, k=1),
        # the pruned field of the benchmark's second leg, at a quarter of its size
        dict(name="pruned_heldout_4m", path="pruned", scene="heldout", n=4_000_000, k=1),
        # filtering outliers from a scene that is kept open
        dict(name="update_csg_1m", path="update", scene="csg", n=1_000_000, k=1),
        # one captured depth map, coloured
        dict(name="depth_1280x960", path="depth", width=1280, height=960, colors=True),
        # the crust of a 4M-sample scene has about this many triangles and few holes
        dict(name="post_300k_triangles", path="post", n=152_000, holes=24, isles=30),
        # training: the batch size of pruner.train
        dict(name="train_batch_8192", path="train", n=8_192),
        # one pass over the leaves of a 4M-sample scene
        dict(name="infer_2m_leaves", path="infer", n=2_000_003),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["crust", "crust", "crust", "crust", "crust", "pruned", "update", "depth", "post", "train",
                       "infer"])
    if path == "crust":
        scene = rng.choice(["sphere", "cluttered", "csg", "csg", "heldout"])
        api = "python" if scene == "sphere" else rng.choice(["host", "device", "python"])
        top = {"sphere": 250_000, "cluttered": 1_000_000, "csg": 4_000_000, "heldout": 12_000_000}[scene]
        if api == "python":
            top = min(top, 2_000_000)
        return dict(path=path, api=api, scene=scene, n=_log_int(rng, 3_000, top), k=rng.choice([1, 1, 2, 3]) if
                    scene == "cluttered" else 1)
    if path == "pruned":
        return dict(path=path, scene=rng.choice(["csg", "heldout"]), n=_log_int(rng, 30_000, 4_000_000), k=1)
    if path == "update":
        return dict(path=path, scene=rng.choice(["csg", "cluttered"]), n=_log_int(rng, 30_000, 1_500_000), k=1)
    if path == "depth":
        w = _log_int(rng, 97, 1_600)
        return dict(path=path, width=w, height=max(2, (w * 3) // 4 + rng.randint(-1, 1)),
                    colors=rng.choice([True, False]))
    if path == "post":
        return dict(path=path, n=_log_int(rng, 3_000, 400_000), holes=rng.randint(0, 40), isles=rng.randint(0, 60))
    if path == "train":
        return dict(path=path, n=_log_int(rng, 500, 65_536))
    return dict(path=path, n=_log_int(rng, 3_000, 8_000_000))


# -------------------------------------------------------------------- inputs


def _scene(case, seed):
    """A scenes.DeviceScene (or scenes.Scene for the sphere) of the case."""
    n, kind = case["n"], case["scene"]
    if kind == "sphere":
        # every stride-th pixel in both directions; 250k samples at stride 3
        stride = max(3, int(math.sqrt(9 * 250_000 / n)))
        sc = scenes.sphere_scene(seed=seed, stride=stride)
        keep = np.sort(np.random.default_rng(seed).choice(sc.n, size=min(n, sc.n), replace=False))
        sc = sc.subset(keep)
    elif kind == "csg":
        sc = scenes.csg_scene_device(seed=seed, n_target=n)
    elif kind == "heldout":
        # the benchmark's held-out geometry and cameras, another capture's noise
        rng = np.random.default_rng(1000 + 999)
        prims = scenes._random_csg_prims(rng, int(rng.integers(3, 9)))
        cams = scenes._random_cams(rng, int(rng.integers(64, 161)), 1.5, 8.0)
        sc = scenes.render_device(prims, cams, 2200, 1650, 1650.0, 0.005, 8.0, seed=seed, target=n, name="heldout")
    else:
        # the benchmark's cluttered capture at a resolution that suits the count
        s = min(1.0, math.sqrt(n / 4_000_000))
        sc = scenes.cluttered_scene_device(seed=seed, n_target=n, width=int(1920 * s) + 1, height=int(1080 * s) + 1,
                                           f=1400.0 * s, n_cams=100)
    if case["k"] > 1:
        # more cameras that saw a sample; a third of the extra slots is empty
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        extra = torch.randint(0, sc.cams.shape[0], (sc.n, case["k"] - 1), generator=gen, device="cuda",
                              dtype=torch.int32)
        empty = torch.rand(extra.shape, generator=gen, device="cuda") < 1.0 / 3.0
        extra[empty] = -1   # 0xFFFFFFFF: no camera
        sc.links = torch.cat([sc.links, extra], 1).contiguous()
    return sc


def _device_view(dev):
    return core.tsr_samples_view(dev["pos"].shape[0], dev["links"].shape[1],
                                 *[dev[k].data_ptr() for k in ("pos", "nrm", "scale", "conf", "links")])


def _arrays(sc):
    return dict(pos=sc.pos, nrm=sc.nrm, scale=sc.scale, conf=sc.conf, links=sc.links)


def _on_device(sc):
    if isinstance(sc.pos, torch.Tensor):
        return _arrays(sc)
    a = _arrays(sc)
    a["links"] = a["links"].view(np.int32)
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()}


class _Surface:
    """Pinned host buffers for a surface, which the program keeps: room for the
    largest one that inputs of its size give, zeros where nothing is written."""

    def __init__(self, cells, vertices, triangles, fields):
        kind = {"cases": (cells, torch.uint8), "positions": (3 * vertices, torch.float64),
                "normals": (3 * vertices, torch.float64), "colors": (3 * vertices, torch.float64),
                "scales": (vertices, torch.float64), "edge_keys": (2 * vertices, torch.int32),
                "triangles": (3 * triangles, torch.int32), "pixel_to_vertex": (cells, torch.int32)}
        self.b = {k: torch.zeros(kind[k][0], dtype=kind[k][1], pin_memory=True) for k in fields}
        self.np = {k: v.numpy() for k, v in self.b.items()}
        self.room = (cells, vertices, triangles)

    def _fits(self, cells, vertices, triangles):
        if cells > self.room[0] or vertices > self.room[1] or triangles > self.room[2]:
            raise ValueError("a surface of %d cells, %d vertices, %d triangles: room for %r" %
                             (cells, vertices, triangles, self.room))

    def take(self, mesh):
        """A core.DualMarchingCells' arrays."""
        nv, nt = mesh.positions.shape[0], mesh.triangles.shape[0]
        self._fits(mesh.cases.shape[0], nv, nt)
        for k in self.np:
            x = getattr(mesh, k).reshape(-1)
            self.np[k][:x.shape[0]] = x.view(np.int32) if x.dtype == np.uint32 else x
        return dict(self.b, counts=np.array([nv, nt]))

    def read(self, mesh, cells):
        """A tsr_mesh's arrays through the C ABI."""
        mc = core.tsr_mesh_counts()
        core._check(core.lib.tsr_mesh_get_counts(mesh, ctypes.byref(mc)))
        self._fits(cells, mc.vertices, mc.triangles)
        p = {k: _ptr(v) for k, v in self.b.items()}
        core._check(core.lib.tsr_mesh_copy(mesh, p.get("cases"), p["positions"], p["scales"], p.get("edge_keys"),
                                           p["triangles"]))
        if "normals" in p and mc.vertices:
            core._check(core.lib.tsr_mesh_copy_normals(mesh, p["normals"]))
        if "colors" in p and mc.vertices:
            core._check(core.lib.tsr_mesh_copy_colors(mesh, p["colors"]))
        if "pixel_to_vertex" in p:
            core._check(core.lib.tsr_mesh_copy_pixel_map(mesh, p["pixel_to_vertex"]))
        return dict(self.b, counts=np.array([mc.vertices, mc.triangles]))


def _crust_surface(n):
    # Few samples on high-resolution images lie far apart, and each is the end
    # of a path of its own in the tree; the counts grow like the square root.
    # The raw crust has no normals, and the post-processed ones are left out: a
    # crust's vertices lie on leaf centres, many triangles have no area, and
    # where a vertex's weighted normals cancel the order of the sum decides.
    r = math.sqrt(n)
    return _Surface(min(int(10_000 * r), 14_000_000), min(int(3_500 * r), 3_000_000), min(int(7_400 * r), 6_300_000),
                    ("cases", "positions", "scales", "edge_keys", "triangles"))


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _damaged_surface(n, holes, isles, seed):
    """A wavy torus grid of about n vertices, triangles cut away inside `holes`
    discs, and `isles` small patches beside it."""
    rng = np.random.default_rng(seed)
    a = max(8, int(math.sqrt(n)))
    b = max(8, n // a)
    u, v = np.meshgrid(np.arange(a) * (2 * math.pi / a), np.arange(b) * (2 * math.pi / b), indexing="ij")
    r = 0.3 + 0.01 * np.sin(7 * u) * np.cos(5 * v) + rng.normal(0, 0.02 / a, u.shape)
    pos = np.stack([(1 + r * np.cos(v)) * np.cos(u), (1 + r * np.cos(v)) * np.sin(u), r * np.sin(v)], -1)
    idx = np.arange(a * b).reshape(a, b)
    i00, i10 = idx, np.roll(idx, -1, 0)
    i01, i11 = np.roll(idx, -1, 1), np.roll(np.roll(idx, -1, 0), -1, 1)
    tri = np.stack([np.stack([i00, i10, i11], -1), np.stack([i00, i11, i01], -1)], 2).reshape(-1, 3)
    pos = pos.reshape(-1, 3)
    centre = pos[tri].mean(1)
    gone = np.zeros(tri.shape[0], bool)
    for c in rng.choice(tri.shape[0], holes, replace=False):
        gone |= np.linalg.norm(centre - centre[c], axis=1) < rng.uniform(2.0, 9.0) * 2.0 / a
    tri = tri[~gone]
    P, T = [pos], [tri]
    base = pos.shape[0]
    for k in range(isles):   # strips of 4 to 40 vertices
        m = int(rng.integers(2, 21))
        x = np.arange(m) * 0.01
        p = np.concatenate([np.stack([x, 0 * x, 0 * x], 1), np.stack([x, 0 * x + 0.01, 0 * x], 1)]) + \
            rng.normal(0, 1, 3) + np.array([0, 0, 3.0])
        q = np.arange(m - 1)
        t = np.concatenate([np.stack([q, q + 1, q + m], 1), np.stack([q + 1, q + m + 1, q + m], 1)])
        P.append(p)
        T.append(t + base)
        base += 2 * m
    return np.concatenate(P), np.concatenate(T).astype(np.uint32)


def _depth_view(case, seed):
    w, h = case["width"], case["height"]
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 2 * math.pi)
    prims = [scenes.Sphere([0, 0, 0], 1.0), scenes.Box([-2.2, -2.2, -1.6], [2.2, 2.2, -1.5])]
    v = scenes.depth_views(prims, [[3 * math.cos(a), 3 * math.sin(a), 0.4]], w, h, 600.0 * w / 1280, 0.001, rng)[0]
    v["depths"][rng.random(v["depths"].shape) < 0.01] = -1.0   # pixels without a depth
    v["colors"] = rng.random((h, w, 3)) if case["colors"] else None
    return v


def _mlp_rows(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, core.MLP_FEATURES), generator=gen, device="cuda")
    y = (torch.rand((n, core.MLP_OUTPUTS), generator=gen, device="cuda") <
         torch.tensor([0.4, 0.2], device="cuda")).float()
    theta = torch.from_numpy(pruner.he_init(seed)).cuda()
    theta += 0.01 * torch.randn(theta.shape, generator=gen, device="cuda")   # biases of a network in training
    return x, y, theta


POS_WEIGHT = (1.5, 4.0)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    s.params = core.params_default()
    path = case["path"]
    if path == "crust":
        sc = _scene(case, seed)
        s.cams = core.Cameras(sc.cams)
        s.out = _crust_surface(case["n"])
        if case["api"] == "python":
            s.samples = core.Samples.from_scene(sc.host() if hasattr(sc, "host") else sc)
        else:
            s.dev = _on_device(sc)
            s.view = _device_view(s.dev)
            if case["api"] == "host":
                s.host = {k: _pinned(v.shape, v.dtype).copy_(v) for k, v in s.dev.items()}
                s.reordered = {k: _pinned(v.shape, v.dtype) for k, v in s.dev.items()}
                s.view = _device_view(s.host)
                s.dev = None
    elif path in ("pruned", "update"):
        sc = _scene(case, seed)
        s.cams = core.Cameras(sc.cams)
        s.tree = core.Tree(core.Samples.from_scene(sc.host()), s.params, reorder_samples=False)
        s.out = _crust_surface(case["n"])
        s.occupancy = _pinned(s.out.room[0], torch.float64)
        if path == "pruned":
            s.pruner = core.Pruner.load()
        else:
            s.again = _crust_surface(case["n"])
            s.occ = core.Occupancy(s.tree, s.cams, s.params)
            n = s.tree.sample_count
            s.chosen = np.sort(np.random.default_rng(seed).choice(n, size=max(1, n // 100), replace=False))
    elif path == "depth":
        s.v = _depth_view(case, seed)
        px = case["width"] * case["height"]
        s.depths = _pinned((px,), torch.float64).copy_(torch.from_numpy(s.v["depths"].reshape(-1)))
        s.colors = None
        if case["colors"]:
            s.colors = _pinned((3 * px,), torch.float64).copy_(torch.from_numpy(s.v["colors"].reshape(-1)))
        s.mvs, s.mws = (np.ascontiguousarray(s.v[k], np.float64) for k in ("hps_to_ray_vs", "hps_to_ray_ws"))
        s.center = np.ascontiguousarray(s.v["center"], np.float64)
        s.out = _Surface(px, px, 2 * px, ("positions", "normals", "colors", "scales", "triangles", "pixel_to_vertex"))
    elif path == "post":
        pos, tri = _damaged_surface(case["n"], case["holes"], case["isles"], seed)
        s.pos = _pinned(pos.shape, torch.float64).copy_(torch.from_numpy(pos))
        s.tri = _pinned(tri.shape, torch.int32).copy_(torch.from_numpy(tri.view(np.int32)))
        s.out = _Surface(0, 2 * case["n"], 4 * case["n"], ("positions", "normals", "scales", "triangles"))
    else:
        s.x, s.y, s.theta = _mlp_rows(case["n"], seed)
        s.grads, s.loss = torch.zeros_like(s.theta), torch.zeros(1, device="cuda")
        s.logits = torch.empty((case["n"], core.MLP_OUTPUTS), device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()   # the renderer's temporaries go back to the device
    return s


# ---------------------------------------------------------------------- runs


def _run_crust_python(s):
    tree = core.Tree(s.samples, s.params, reorder_samples=False)
    occ = core.Occupancy(tree, s.cams, s.params)
    return s.out.take(occ.extractCrust(min_isle_size=1000))


def _run_crust_c(s):
    lib, chk, ref = core.lib, core._check, ctypes.byref
    st = _stream()
    on_device = s.case["api"] == "device"
    tree, occ, mesh = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    out = {}
    try:
        build = lib.tsr_tree_build_device if on_device else lib.tsr_tree_build
        chk(build(ref(s.view), ref(s.params), st, ref(tree)))
        if not on_device:
            chk(lib.tsr_tree_copy_samples(tree, *[_ptr(s.reordered[k]) for k in
                                                  ("pos", "nrm", "scale", "conf", "links")]))
            out.update(s.reordered)
        chk(lib.tsr_occupancy_compute(tree, ref(s.cams.view()), ref(s.params), 0, st, ref(occ)))
        chk(lib.tsr_dmc_extract(tree, occ, st, ref(mesh)))
        tc = core.tsr_tree_counts()
        chk(lib.tsr_tree_get_counts(tree, ref(tc)))
        out.update(s.out.read(mesh, tc.dual_cells))
        return out
    finally:
        if mesh:
            lib.tsr_mesh_free(mesh)
        if occ:
            lib.tsr_occupancy_free(occ)
        if tree:
            lib.tsr_tree_free(tree)


def _surface_of(occ, out):
    """The surface of a kept field, read into kept buffers."""
    mesh = ctypes.c_void_p()
    core._check(core.lib.tsr_dmc_extract(occ.tree.handle, occ.handle, None, ctypes.byref(mesh)))
    try:
        return out.read(mesh, occ.tree.counts["dual_cells"])
    finally:
        core.lib.tsr_mesh_free(mesh)


def _values_of(occ, out):
    core._check(core.lib.tsr_occupancy_copy(occ.handle, core.FIELDS["occupancy"], _ptr(out)))
    return out


def run(state):
    s = state
    lib, chk, ref = core.lib, core._check, ctypes.byref
    path = s.case["path"]
    if path == "crust":
        return _run_crust_python(s) if s.case["api"] == "python" else _run_crust_c(s)
    if path == "pruned":
        occ = core.Occupancy(s.tree, s.cams, s.params, pruner=s.pruner)
        return dict(surface=_surface_of(occ, s.out), occupancy=_values_of(occ, s.occupancy))
    if path == "update":
        s.occ.eraseSamples(s.chosen, s.cams, s.params)
        without = _surface_of(s.occ, s.out)
        s.occ.addSamples(s.chosen, s.cams, s.params)
        return dict(without=without, again=_surface_of(s.occ, s.again), occupancy=_values_of(s.occ, s.occupancy))
    if path in ("depth", "post"):
        mesh = ctypes.c_void_p()
        try:
            if path == "depth":
                chk(lib.tsr_depth_triangulate(_ptr(s.depths), s.case["width"], s.case["height"],
                                              s.mvs.ctypes.data_as(ctypes.c_void_p),
                                              s.mws.ctypes.data_as(ctypes.c_void_p),
                                              s.center.ctypes.data_as(ctypes.c_void_p),
                                              None if s.colors is None else _ptr(s.colors), _stream(), ref(mesh)))
            else:
                chk(lib.tsr_mesh_create(_ptr(s.pos), None, s.pos.shape[0], _ptr(s.tri), s.tri.shape[0], _stream(),
                                        ref(mesh)))
                chk(lib.tsr_mesh_postprocess(mesh, 1000, None))
            return s.out.read(mesh, 0)
        finally:
            if mesh:
                lib.tsr_mesh_free(mesh)
    if path == "train":
        s.grads.zero_()
        s.loss.zero_()
        chk(lib.tsr_mlp_train_batch(_ptr(s.x), _ptr(s.y), s.case["n"], _ptr(s.theta), _ptr(s.grads), _ptr(s.loss),
                                    POS_WEIGHT[0], POS_WEIGHT[1], _stream()))
        return dict(grads=s.grads, loss=s.loss)
    chk(lib.tsr_mlp_infer_bf16(_ptr(s.x), s.case["n"], _ptr(s.theta), _ptr(s.logits), _stream()))
    return s.logits


# ---------------------------------------------------------------------- work


def work(case):
    """Compulsory bytes and operations of one pass.

    The volumetric core per unit: a sample is read by the build and written in
    tree order, then read once per cone pass; nodes, leaves and dual cells are
    written once and read once per pass that needs them.  Over the scenes and
    sizes here a tree has about 1500 sqrt(n) leaves, 1.14 nodes and 1.35 dual
    cells per leaf, and a link is accepted by about 0.15 sqrt(n), at most 400,
    leaves (about 40 operations each).
    """
    path, n = case["path"], case.get("n", 0)
    if path in ("crust", "pruned", "update"):
        links = n * case["k"]
        nl = 1500.0 * math.sqrt(n)
        nn, nc = 1.14 * nl, 1.35 * nl
        priors = nn * 16 + nl * (16 + 8)
        field = 2 * (n * 64 + links * 4) + priors + nl * (8 * 6 + 16)
        mesh = nc * (32 + 1) + nl * 8 + 0.3 * nl * 60
        pairs = min(400.0, 0.15 * math.sqrt(n)) * links
        if path == "crust":
            tree = n * (64 + 4 * case["k"]) * 2 + nn * 40 + nl * 60 + nc * 32
            return {"bytes": tree + field + mesh, "flops": 40 * pairs}
        if path == "pruned":
            return {"bytes": field + mesh + nl * 8, "flops": 40 * pairs + nl * 2 * (10 * 64 + 64 * 64 + 128)}
        # two updates of 1 % of the links, each with every prior and value again
        return {"bytes": 2 * (priors + nl * 8 * 6 + mesh) + nl * 8, "flops": 2 * 0.01 * 40 * pairs}
    if path == "depth":
        px = case["width"] * case["height"]
        nv, nt = 0.35 * px, 0.7 * px
        return {"bytes": px * (8 + 4 + (24 if case["colors"] else 0)) + nv * 80 + nt * 12, "flops": nt * 300.0}
    if path == "post":
        return {"bytes": n * (24 * 3 + 16) + 2 * n * 24, "flops": 2 * n * 200.0}
    macs = 10 * 64 + 64 * 64 + 64 * 2
    if path == "train":
        return {"bytes": n * 48 + 3 * core.MLP_PARAMS * 4, "flops": 6.0 * n * macs}
    return {"bytes": n * 48 + core.MLP_PARAMS * 4, "flops": 2.0 * n * macs}


# --------------------------------------------------------------------- exact


def _split(theta):
    t = theta.double()
    o = 0
    parts = []
    for shape in ((10, 64), (64,), (64, 64), (64,), (64, 2), (2,)):
        m = math.prod(shape)
        parts.append(t[o:o + m].reshape(shape))
        o += m
    return parts


def _forward64(x, parts):
    w1, b1, w2, b2, w3, b3 = parts
    return torch.relu(torch.relu(x.double() @ w1 + b1) @ w2 + b2) @ w3 + b3


def _unit(v):
    l = np.linalg.norm(v, axis=-1, keepdims=True)
    return np.divide(v, l, out=v.copy(), where=l > 0)


def _exact_depth(case, seed):
    v = _depth_view(case, seed)
    d, mvs, mws = v["depths"], v["hps_to_ray_vs"], v["hps_to_ray_ws"]
    h, w = d.shape
    ys, xs = np.mgrid[0:h, 0:w]
    hps = np.stack([xs, ys, np.ones_like(xs)], -1).astype(float)
    foot = mvs[0, 0] * d / np.linalg.norm(hps @ mvs, axis=-1)
    pix = np.arange(h * w).reshape(h, w)
    block = lambda a: np.stack([a[:-1, :-1], a[:-1, 1:], a[1:, :-1], a[1:, 1:]], -1).reshape(-1, 4)  # noqa: E731
    bd, bf, bp = block(d), block(foot), block(pix)
    code = (bd > 0) @ np.array([1, 2, 4, 8])
    first = np.full(code.shape, -1)
    second = np.full(code.shape, -1)
    for k, m in enumerate((7, 11, 13, 14)):
        first[code == m] = k
    full = code == 15
    one = np.abs(bd[:, 0] - bd[:, 3]) < np.abs(bd[:, 1] - bd[:, 2])
    first[full] = np.where(one[full], 1, 0)
    second[full] = np.where(one[full], 2, 3)
    kinds = np.array([[0, 2, 1], [0, 3, 1], [0, 2, 3], [1, 2, 3]])
    both = np.stack([first, second], 1)
    rows, slot = np.nonzero(both >= 0)
    corner = kinds[both[rows, slot]]
    cd, cf = np.take_along_axis(bd[rows], corner, 1), np.take_along_axis(bf[rows], corner, 1)
    ok = np.ones(rows.size, bool)
    for e in range(3):
        a, b = e, (e + 1) % 3
        near = np.where(cd[:, a] < cd[:, b], cf[:, a], cf[:, b])
        diagonal = corner[:, a] + corner[:, b] == 3
        ok &= ~(np.abs(cd[:, a] - cd[:, b]) > near * np.where(diagonal, 5.0 * math.sqrt(2.0), 5.0))
    corners = np.take_along_axis(bp[rows], corner, 1)[ok].reshape(-1)
    used, at = np.unique(corners, return_index=True)
    used = used[np.argsort(at)]   # a pixel's vertex is numbered when a corner first names it
    num = np.full(h * w, -1)
    num[used] = np.arange(used.size)
    tri = num[corners].reshape(-1, 3)
    pos = v["center"] + _unit((hps.reshape(-1, 3)[used]) @ mws) * d.reshape(-1)[used][:, None]
    p = pos[tri]
    n = _unit(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]))
    nrm = np.zeros_like(pos)
    for k in range(3):
        a, b = _unit(p[:, (k + 1) % 3] - p[:, k]), _unit(p[:, (k + 2) % 3] - p[:, k])
        ang = np.arccos(np.clip((a * b).sum(1), -1, 1))
        for j in range(3):
            nrm[:, j] += np.bincount(tri[:, k], weights=n[:, j] * ang, minlength=pos.shape[0])
    e = np.concatenate([tri[:, [0, 1]], tri[:, [1, 2]], tri[:, [2, 0]]])
    key = np.unique(np.minimum(e[:, 0], e[:, 1]) * np.int64(pos.shape[0]) + np.maximum(e[:, 0], e[:, 1]))
    a, b = key // pos.shape[0], key % pos.shape[0]
    dist = np.linalg.norm(pos[a] - pos[b], axis=1)
    tot = np.bincount(a, dist, pos.shape[0]) + np.bincount(b, dist, pos.shape[0])
    cnt = np.bincount(a, minlength=pos.shape[0]) + np.bincount(b, minlength=pos.shape[0])
    colors = np.full((pos.shape[0], 3), 0.5) if v["colors"] is None else v["colors"].reshape(-1, 3)[used]

    def room(x, c):   # the kept buffers have room for a vertex at every pixel
        return np.concatenate([x.reshape(-1), np.zeros(c * h * w - x.size)])

    return dict(positions=room(pos, 3), normals=room(_unit(nrm), 3), colors=room(colors, 3), scales=room(tot / cnt, 1),
                triangles=None, pixel_to_vertex=None, counts=None)


def exact(case, seed):
    path = case["path"]
    if path == "depth":
        return _exact_depth(case, seed)
    if path in ("train", "infer"):
        x, y, theta = _mlp_rows(case["n"], seed)
        parts = _split(theta)
        if path == "infer":
            return torch.cat([_forward64(c, parts) for c in x.split(1 << 20)])
        for p in parts:
            p.requires_grad_(True)
        z = _forward64(x, parts)
        t = y.double()
        weight = torch.where(t > 0.5, torch.tensor(POS_WEIGHT, dtype=torch.float64, device="cuda"), torch.ones_like(t))
        loss = (weight * torch.nn.functional.binary_cross_entropy_with_logits(z, t, reduction="none")).sum()
        g = torch.autograd.grad(loss, parts)
        return dict(grads=torch.cat([v.reshape(-1) for v in g]), loss=loss.detach().reshape(1))
    # The surface: the tree's sampling nodes depend on each other in the order
    # of the samples, which plain Python replays in minutes, not seconds.  The
    # filled holes likewise follow a sequential search.
    return None
