"""The work that programs give this library, as timed cases.

Each case is one call (or the few calls that belong together) of the Python
surface over the C ABI, on the scenes that the benchmark and the tests use:
sphere unions, noise terrains and displaced icospheres, seeded.  `listed()`
names the cases, `draw()` gives others of the same ranges, `prepare()` makes
what a program holds before the call, `run()` makes the call once and returns
everything it computes, `work()` gives the bytes and operations it cannot do
without, and `exact()` the results in 64 bits where such results exist.
Where a result's size depends on the geometry (an octree's words, per-leaf
arrays), the geometry comes from the case's `shape` seed and the seed gives
the rest: payloads, colours, cameras, parameters.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sparse-voxel-octrees_gb300")
GIB = 1 << 30


def _package():
    """The package, whose folder's name is not an identifier, as svo_gb300."""
    if "svo_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("svo_gb300", os.path.join(PKG, "__init__.py"),
                                                      submodule_search_locations=[PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["svo_gb300"] = mod
        spec.loader.exec_module(mod)
    import svo_gb300.scenes as scenes
    return sys.modules["svo_gb300"], scenes


def listed():
    return [
        # One ray picked against a loaded octree, as a program written for the
        # reference's VoxelOctree::raymarch does for a mouse position or a
        # line of sight: the smallest call, all latency.
        {"name": "pick_ray", "kind": "host_rays", "scene": "sphere", "side": 256, "n": 1},
        # A preview or a tile of a viewport: the smallest view of the batched
        # workload's range.
        {"name": "view_256", "kind": "view", "scene": "sphere", "side": 128, "width": 256, "height": 256},
        # The benchmark's large traversal, one of its cameras: a full frame of
        # primary rays from device memory over a 2048^3 terrain.
        {"name": "view_1080p_2048", "kind": "view", "scene": "terrain", "side": 2048, "width": 1920, "height": 1080},
        # One shadow ray per surface point toward a light: incoherent rays
        # that are no image, hit flags only.
        {"name": "shadow_rays", "kind": "shadow", "scene": "terrain", "side": 1024, "n": 830000},
        # Many objects at uneven depths and resolutions in one graph launch.
        {"name": "batch_12", "kind": "batch", "views": 12, "max_depth": 10, "shape": 3},
        # The viewer's frame at its window size, beam prepass included.
        {"name": "frame_720p", "kind": "frame", "scene": "terrain", "side": 1024, "width": 1280, "height": 720,
         "stride": 1},
        # A CPU program's view: rays and results in page-locked host memory.
        {"name": "host_view_768", "kind": "host_view", "scene": "sphere", "side": 256, "width": 1024, "height": 768},
        # One optimisation step of the leaf-shading workload: forward, fused
        # adjoint of the L2 loss, Adam over the touched leaves' records.
        {"name": "shading_step", "kind": "train", "side": 256, "spheres": 80, "views": 12, "width": 512,
         "height": 512, "shape": 7},
        # Forward and adjoint for a caller's own loss: dL/drgb given, the
        # parameter arrays apart, the adjoint tracing again to save the hit
        # buffer, a ragged image.
        {"name": "shading_retrace", "kind": "adjoint", "side": 256, "spheres": 48, "views": 3, "width": 333,
         "height": 251, "shape": 0},
        # An octree from a dense voxel grid in device memory (a simulation's or
        # a reconstruction's output), at the shading workload's size.
        {"name": "build_512", "kind": "build", "scene": "sphere", "w": 512, "h": 512, "d": 512, "mem": GIB,
         "view": False, "shape": 7},
        # An edited small volume, rebuilt and shown: ragged sides, the build
        # and the new octree's first view.
        {"name": "edit_and_view", "kind": "build", "scene": "sphere", "w": 200, "h": 131, "d": 177, "mem": GIB,
         "view": True, "shape": 0},
        # A triangle mesh voxelized at 1024^3 and built into an octree: the
        # benchmark's mesh (327,680 triangles, 16 sub-blocks, 1 GiB).
        {"name": "mesh_1024", "kind": "mesh", "level": 7, "side": 1024, "threads": 16, "mem": GIB,
         "shape": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, lo, hi):
    """Width and height of lo to hi pixels at about 16:9, odd sizes among them."""
    pix = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    w = max(8, min(1920, int((pix * rng.uniform(1.2, 1.9)) ** 0.5)))
    return w, max(8, min(1080, int(pix / w)))


def draw(rng):
    kind = rng.choice(["host_rays", "view", "shadow", "batch", "frame", "host_view", "train", "adjoint", "build",
                       "build", "mesh"])
    scene = rng.choice(["sphere", "terrain"])
    side, shape = 1 << rng.randint(7, 10), rng.randrange(1 << 20)
    if kind == "host_rays":
        return {"kind": kind, "scene": scene, "side": side, "n": _log_int(rng, 1, 60000)}
    if kind == "shadow":
        return {"kind": kind, "scene": scene, "side": side, "n": _log_int(rng, 500, 830000)}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(3, 12), "max_depth": rng.randint(8, 10), "shape": shape}
    if kind == "frame":
        w, h = _image(rng, 320 * 180, 1280 * 720)
        return {"kind": kind, "scene": scene, "side": side, "width": w, "height": h, "stride": rng.choice([1, 1, 3])}
    if kind in ("view", "host_view"):
        w, h = _image(rng, 64 * 64, 1920 * 1080 if kind == "view" else 1024 * 768)
        return {"kind": kind, "scene": scene, "side": side, "width": w, "height": h}
    if kind in ("train", "adjoint"):
        w, h = _image(rng, 96 * 96, 512 * 512)
        return {"kind": kind, "side": 1 << rng.randint(7, 8), "spheres": rng.randint(20, 80),
                "views": rng.randint(1, 12 if kind == "train" else 6), "width": w, "height": h, "shape": shape}
    if kind == "build":
        lo, hi = rng.choice([(24, 128), (100, 256), (200, 512)])
        return {"kind": kind, "scene": scene, "w": _log_int(rng, lo, hi), "h": _log_int(rng, lo, hi),
                "d": _log_int(rng, lo, hi), "mem": rng.choice([GIB, 16 << 20]), "view": rng.random() < 0.5,
                "shape": shape}
    return {"kind": kind, "level": rng.randint(3, 7), "side": _log_int(rng, 64, 1024), "threads": rng.randint(1, 16),
            "mem": rng.choice([GIB, 128 << 20]), "shape": shape}


# ---- inputs


def _grid(scenes, scene, side, seed, spheres=None):
    if scene == "sphere":
        return scenes.gpu_sphere_scene(side, spheres or 48, seed)
    return scenes.gpu_terrain_scene(side, spheres or 200, seed)


def _tree(svo, scenes, case, seed):
    side = case["side"]
    grid = _grid(scenes, case.get("scene", "sphere"), side, seed, case.get("spheres"))
    return svo.VoxelOctree(svo.VoxelData(grid, max(8 * GIB, 4 * side ** 3))), grid


def _camera(scenes, scene, center, seed):
    """An orbit camera; a terrain's is nearer, as the benchmark's are."""
    if scene == "sphere":
        return scenes.orbit_cameras(1, seed, center, radius=2.0)[0]
    return scenes.orbit_cameras(1, seed, center, radius=1.25, radius_hi=2.0, pitch=45.0)[0]


def _dev(n, dtype=torch.float32):
    return torch.empty(n, dtype=dtype, device="cuda")


def _image_out(n):
    # what the reference computes per pixel: t, the leaf word and the viewer's 8-bit colour
    return {"t": _dev(n), "word": _dev(n, torch.int32), "rgba8": _dev(n, torch.int32)}


def _pick_rays(center, n, seed):
    """Unit rays from an orbit toward random points of the volume's middle."""
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(n, 3))
    o = 1.0 + center + 2.0 * o / np.linalg.norm(o, axis=1, keepdims=True)
    d = 1.0 + center + rng.uniform(-0.25, 0.25, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _shading(svo, scenes, case, seed, stride):
    """Octree, rays, lights, targets, parameters and buffers of the shading workload."""
    tree, _ = _tree(svo, scenes, case, case["shape"])
    W, H, V = case["width"], case["height"], case["views"]
    cams = scenes.orbit_cameras(V, seed, tree.center(), radius=2.0)
    R = V * W * H
    rays = _dev((R, 6))
    for i, c in enumerate(cams):
        scenes.gpu_camera_rays(c, W, H, out=rays[i * W * H:(i + 1) * W * H])
    lights = torch.from_numpy(np.stack([scenes.headlight(c) for c in cams]).astype(np.float32)).cuda()
    # the true colours: a noise field at the hit points
    t, leaf = _dev(R), _dev(R, torch.int32)
    tree.trace(rays, out={"t": t, "leaf": leaf})
    hit = leaf != -1
    target = torch.zeros((R, 3), device="cuda")
    p = rays[hit, :3] + t[hit, None] * rays[hit, 3:]
    target[hit] = torch.stack([scenes.noise3(p, seed % 1000 + k) for k in range(3)], 1)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nw = tree.num_words()
    s = {"tree": tree, "rays": rays, "lights": lights, "target": target, "view": (W, H, V), "rgb": _dev((R, 3)),
         "leaf": _dev(R, torch.int32), "scale": 2.0 / (3 * R), "hits": leaf}
    if stride == 8:  # one record a leaf: colour, normal, two floats unused
        rec = torch.zeros((nw, 8), device="cuda")
        rec[:, :6] = torch.rand((nw, 6), generator=gen, device="cuda")
        rec.grad = torch.zeros_like(rec)
        s.update(rec=rec, leaves=svo.LeafSet(nw), loss=torch.zeros(1, dtype=torch.float64, device="cuda"))
        s["opt"] = svo.LeafAdam([rec], lr=1e-2, leaves=s["leaves"], width=8)
    else:
        s.update(p_rgb=torch.rand((nw, 3), generator=gen, device="cuda"),
                 p_n=torch.rand((nw, 3), generator=gen, device="cuda"), g_rgb=torch.zeros((nw, 3), device="cuda"),
                 g_n=torch.zeros((nw, 3), device="cuda"), d_rgb=torch.randn((R, 3), generator=gen, device="cuda"))
    return s


def prepare(case, seed):
    svo, scenes = _package()
    kind = case["kind"]
    if kind in ("view", "host_view"):
        tree, _ = _tree(svo, scenes, case, seed)
        cam = _camera(scenes, case["scene"], tree.center(), seed)
        W, H = case["width"], case["height"]
        rays = scenes.gpu_camera_rays(cam, W, H)
        s = {"kind": kind, "tree": tree, "rays": rays, "size": (W, H), "light": scenes.headlight(cam)}
        if kind == "view":
            s["out"] = _image_out(W * H)
            return s
        s["keep"] = [rays.cpu().pin_memory()] + [torch.empty(W * H, dtype=d).pin_memory()
                                                 for d in (torch.float32, torch.int32, torch.int32)]
        host = [x.numpy() for x in s["keep"]]
        s["rays"], s["out"] = host[0], dict(zip(("t", "word", "rgba8"), host[1:]))
        return s
    if kind == "host_rays":
        tree, _ = _tree(svo, scenes, case, seed)
        return {"kind": kind, "tree": tree, "rays": _pick_rays(tree.center(), case["n"], seed)}
    if kind == "shadow":
        tree, _ = _tree(svo, scenes, case, seed)
        W, H = 1280, 720
        cam = _camera(scenes, case["scene"], tree.center(), seed)
        rays = scenes.gpu_camera_rays(cam, W, H)
        t, hit = _dev(W * H), _dev(W * H, torch.uint8)
        tree.trace(rays, out={"t": t, "hit": hit})
        # the surface points, ordered by 8x4-pixel tile, as many as asked for
        pix = torch.arange(W * H, device="cuda")
        px, py = pix % W, pix // W
        order = torch.argsort(((py // 4) * ((W + 7) // 8) + px // 8) * 32 + (py % 4) * 8 + px % 8)
        at = order[hit[order] == 1]
        if at.numel() == 0:
            at = order
            t = torch.full_like(t, 2.0)
        n = case["n"]
        at = at[torch.arange(n, device="cuda") * at.numel() // n]
        light = torch.tensor([0.3, 0.8, 0.52], device="cuda")
        light = light / light.norm()
        o = rays[at, :3] + t[at, None] * rays[at, 3:] + (1.5 / case["side"]) * light
        return {"kind": kind, "tree": tree, "rays": torch.cat([o, light.expand_as(o)], 1).contiguous(),
                "out": {"hit": _dev(n, torch.uint8)}}
    if kind == "batch":
        specs, views, total = [], [], 0
        for i, side, gen, W, H in scenes.batched_views(case["views"], case["shape"]):
            side = min(side, 1 << case["max_depth"])
            W, H = min(W, 1280), min(H, 720)
            specs.append((i, side, gen, W, H, total))
            total += W * H
        out = {"t": _dev(total), "leaf": _dev(total, torch.int32), "rgba8": _dev(total, torch.int32)}
        for i, side, gen, W, H, at in specs:
            tree, _ = _tree(svo, scenes, {"scene": gen, "side": side}, case["shape"] + i)
            cam = scenes.orbit_cameras(1, seed + i, tree.center(), radius=2.0)[0]
            views.append({"octree": tree, "width": W, "height": H, "camera": scenes.camera_constants(cam, W, H),
                          "light": scenes.headlight(cam), "out": {k: v[at:at + W * H] for k, v in out.items()}})
        batch = svo.Batch(views)
        # the launch shape that the autotuner finds for the benchmark's batches
        batch.capture_graph(svo.default_config(refill_idle=32, steps_per_round=64, reg_cap=48))
        return {"kind": kind, "batch": batch, "out": out}
    if kind == "frame":
        tree, _ = _tree(svo, scenes, case, seed)
        rng = np.random.default_rng(seed)
        rot, _, pos = scenes.viewer_camera(rng.uniform(0, 360), rng.uniform(-45, 45), rng.uniform(1.25, 2.0),
                                           tree.center())
        W, H = case["width"], case["height"]
        return {"kind": kind, "tree": tree, "rot": rot, "pos": pos, "size": (W, H), "stride": case["stride"],
                "out": torch.empty((H, W), dtype=torch.int32, device="cuda")}
    if kind in ("train", "adjoint"):
        return dict(_shading(svo, scenes, case, seed, 8 if kind == "train" else 3), kind=kind)
    if kind == "build":
        w, h, d = case["w"], case["h"], case["d"]
        side = max(32, 1 << (max(w, h, d) - 1).bit_length())
        grid = _grid(scenes, case["scene"], side, case["shape"])[:d, :h, :w].contiguous()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        full = grid != 0  # other shades in the words' low 7 bits
        grid ^= torch.randint(0, 128, grid.shape, generator=gen, device="cuda", dtype=torch.int32) * full
        grid += (full & (grid == 0)).to(torch.int32)
        s = {"kind": kind, "data": svo.VoxelData(grid, case["mem"]), "tree": None, "rays": None}
        if case["view"]:
            cam = scenes.orbit_cameras(1, seed, np.array([w, h, d]) * 0.5 / side, radius=2.0)[0]
            s.update(rays=scenes.gpu_camera_rays(cam, 640, 480), light=scenes.headlight(cam), out=_image_out(640 * 480))
        return s
    if kind == "mesh":
        pos, faces, _ = scenes.displaced_icosphere(case["level"], case["shape"])
        col = np.random.default_rng(seed).integers(0, 256, pos.shape).astype(np.float32)
        loader = svo.PlyLoader.from_arrays(pos, faces, colors=col)
        return {"kind": kind, "data": svo.VoxelData(loader, case["side"], case["mem"], case["threads"]), "tree": None}
    raise ValueError(kind)


# ---- one pass


class _Words:
    """An octree's resident words, for torch to look at where they are."""

    def __init__(self, tree):
        self.tree = tree
        self.__cuda_array_interface__ = {"shape": (tree.num_words(),), "typestr": "<i4", "version": 2,
                                         "data": (tree.device_words_ptr(), False)}


def run(s):
    svo, _ = _package()
    kind = s["kind"]
    if kind == "view":
        s["tree"].trace_image(s["rays"], *s["size"], light=s["light"], out=s["out"])
        return s["out"]
    if kind == "host_view":
        return s["tree"].trace_image_host(s["rays"], *s["size"], light=s["light"], out=s["out"])
    if kind == "host_rays":
        rays = s["rays"]
        if len(rays) == 1:
            hit, word, t = s["tree"].raymarch(rays[0, :3], rays[0, 3:])
            return {"hit": int(hit), "word": word or 0, "t": np.float32(t if hit else np.inf)}
        return s["tree"].trace_host(rays, outputs=("hit", "word", "t"))
    if kind == "shadow":
        s["tree"].trace(s["rays"], out=s["out"])
        return s["out"]
    if kind == "batch":
        s["batch"].launch_graph()
        return s["out"]
    if kind == "frame":
        return s["tree"].render_frame(s["rot"], s["pos"], *s["size"], n_strips=16, pixel_stride=s["stride"],
                                      out=s["out"])
    if kind == "train":
        rec, g = s["rec"], s["rec"].grad
        common = (s["rays"], *s["view"], s["lights"], rec[:, 0:3], rec[:, 3:6])
        s["loss"].zero_()
        s["tree"].diff_forward(*common, s["rgb"], hit_leaf=s["leaf"], param_stride=8)
        s["tree"].diff_backward_l2(*common, s["rgb"], s["target"], s["scale"], g[:, 0:3], g[:, 3:6],
                                   hit_leaf=s["leaf"], loss_sum=s["loss"], leaves=s["leaves"], param_stride=8)
        s["opt"].step()
        m, v = s["opt"].state[0]
        return {"rgb": s["rgb"], "leaf": s["leaf"], "loss": s["loss"], "params": rec, "exp_avg": m, "exp_avg_sq": v}
    if kind == "adjoint":
        common = (s["rays"], *s["view"], s["lights"], s["p_rgb"], s["p_n"])
        s["g_rgb"].zero_()
        s["g_n"].zero_()
        s["tree"].diff_forward(*common, s["rgb"])
        s["tree"].diff_backward(*common, s["d_rgb"], s["g_rgb"], s["g_n"])
        return {"rgb": s["rgb"], "g_rgb": s["g_rgb"], "g_n": s["g_n"]}
    s["tree"] = svo.VoxelOctree(s["data"])  # replaces the octree of the pass before
    words = torch.as_tensor(_Words(s["tree"]), device="cuda")
    if kind == "build" and s["rays"] is not None:
        s["tree"].trace_image(s["rays"], 640, 480, light=s["light"], out=s["out"])
        return dict(s["out"], words=words)
    return {"words": words}


# ---- what a pass cannot do without


def work(case):
    """Inputs read once, outputs written once; an octree's touched part is left
    out where it depends on the scene.  Operations: about 30 traversal steps
    of 20 operations a ray, about 150 a (voxel, triangle) test."""
    kind = case["kind"]
    step = 600.0
    if kind in ("view", "host_view"):
        n = case["width"] * case["height"]
        return {"bytes": n * (24 + 12), "flops": n * step}
    if kind == "host_rays":
        return {"bytes": case["n"] * (24 + 9), "flops": case["n"] * step}
    if kind == "shadow":
        return {"bytes": case["n"] * (24 + 1), "flops": case["n"] * step}
    if kind == "batch":
        n = case["views"] * 480000  # the mean of the log-uniform sizes, about
        return {"bytes": n * 12, "flops": n * step}
    if kind == "frame":
        n = case["width"] * case["height"]
        return {"bytes": n * 4, "flops": n * step}
    if kind in ("train", "adjoint"):
        n = case["width"] * case["height"] * case["views"]
        # rays twice, dL/drgb or target, colours; half of the rays hit, about
        # four to a leaf: its parameters, gradients and moments
        leaves = n / 8
        if kind == "train":
            return {"bytes": n * (24 + 12 + 4 + 24 + 4 + 24) + leaves * 24 * 8, "flops": n * step}
        return {"bytes": n * (24 + 12 + 24 + 12) + leaves * 24 * 3, "flops": 2 * n * step}
    if kind == "build":
        cells = case["w"] * case["h"] * case["d"]
        # about a quarter of a sphere union's cells and 1 % of a terrain's become words
        words = cells * (0.28 if case["scene"] == "sphere" else 0.012)
        return {"bytes": cells * 4 + words * 4 + (640 * 480 * 36 if case["view"] else 0), "flops": cells}
    tris = 20.0 * 4 ** case["level"]
    voxels = 4.3 * case["side"] ** 2
    return {"bytes": tris * 72 + voxels * 4 * 1.33, "flops": voxels * 6 * 150}


# ---- results in 64 bits


def _march64(occ, rays):
    """t of each ray's first occupied cell in a (d, h, w) occupancy whose
    octree has side max(occ.shape) rounded up to a power of two, by stepping
    from cell to cell; inf where there is none."""
    side = 1 << (max(occ.shape) - 1).bit_length()
    d, h, w = occ.shape
    rays = rays.to(torch.float64)
    dirs = torch.where(rays[:, 3:].abs() < 1e-4, torch.full_like(rays[:, 3:], 1e-4), rays[:, 3:]) * side
    o = (rays[:, :3] - 1.0) * side
    a, b = -o / dirs, (side - o) / dirs
    t = torch.minimum(a, b).amax(1).clamp(min=0.0)
    end = torch.maximum(a, b).amin(1)
    p = o + t[:, None] * dirs
    cell = p.floor().clamp(0, side - 1).to(torch.int64)
    step = torch.where(dirs > 0, 1, -1)
    res = torch.full_like(t, math.inf)
    live = t < end
    size = torch.tensor([w, h, d], device=occ.device)
    for _ in range(3 * side + 3):
        if not bool(live.any()):
            break
        c = torch.minimum(cell.clamp(min=0), size - 1)
        full = live & (cell < size).all(1) & occ[c[:, 2], c[:, 1], c[:, 0]]
        res = torch.where(full, t, res)
        nxt = ((cell + (step > 0)) - o) / dirs
        t_next, axis = nxt.min(1)
        live = live & ~full
        t = torch.where(live, torch.maximum(t, t_next), t)
        cell = cell.scatter_add(1, axis[:, None], step.gather(1, axis[:, None]))
        live = live & ((cell >= 0) & (cell < side)).all(1)
    return res


def _shade64(s, p_rgb, p_n, g=None):
    """The leaf shading of every ray in 64 bits, its squared distance from the
    target, and the adjoint of `g` (dL/drgb) if given or of the L2 loss."""
    W, H, V = s["view"]
    hit = s["hits"] != -1
    leaf = s["hits"][hit].to(torch.int64) & 0xFFFFFFFF
    d = s["rays"][hit, 3:].double()
    view = torch.arange(V, device="cuda").repeat_interleave(W * H)[hit]
    l = s["lights"].double()[view]
    c, p = p_rgb.double()[leaf], p_n.double()[leaf]
    inv = 1.0 / p.norm(dim=1, keepdim=True)
    n = p * inv
    ln, nd = (l * n).sum(1, keepdim=True), (n * d).sum(1, keepdim=True)
    sp = ((l * (d - 2 * nd * n)).sum(1, keepdim=True)).clamp(min=0)
    rgb = torch.zeros((V * W * H, 3), dtype=torch.float64, device="cuda")
    rgb[hit] = c * 0.9 * ln.abs() + 0.2 * sp * sp
    err = rgb - s["target"].double()
    g = (s["scale"] * err if g is None else g.double())[hit]
    gc = torch.zeros((p_rgb.shape[0], 3), dtype=torch.float64, device="cuda")
    gn = torch.zeros_like(gc)
    gc.index_add_(0, leaf, g * 0.9 * ln.abs())
    dn = 0.9 * torch.sign(ln) * (g * c).sum(1, keepdim=True) * l - \
        0.8 * g.sum(1, keepdim=True) * sp * (nd * l + ln * d)
    gn.index_add_(0, leaf, (dn - n * (n * dn).sum(1, keepdim=True)) * inv)
    return rgb, (err * err).sum().reshape(1), gc, gn


def exact(case, seed):
    """The shading cases whole; t of rays and small views by a plain march
    (hit flags, leaf indices, words and packed colours are whole numbers).  A
    large image has none: the traversal is defined in 32 bits, and some rays
    grazing an edge hit in 32 bits and miss in 64."""
    svo, scenes = _package()
    kind = case["kind"]
    if kind == "train":
        s = _shading(svo, scenes, case, seed, 8)
        rec = s["rec"]
        rgb, loss, gc, gn = _shade64(s, rec[:, 0:3], rec[:, 3:6])
        g = torch.cat([gc, gn, torch.zeros((rec.shape[0], 2), dtype=torch.float64, device="cuda")], 1)
        m, v = 0.1 * g, 0.001 * g * g
        p = rec.double() - 1e-2 / (1 - 0.9) * m / (v.sqrt() / (1 - 0.999) ** 0.5 + 1e-8)
        return {"rgb": rgb, "leaf": None, "loss": loss, "params": p, "exp_avg": m, "exp_avg_sq": v}
    if kind == "adjoint":
        s = _shading(svo, scenes, case, seed, 3)
        rgb, _, gc, gn = _shade64(s, s["p_rgb"], s["p_n"], s["d_rgb"])
        return {"rgb": rgb, "g_rgb": gc, "g_n": gn}
    if kind == "host_rays":
        tree, grid = _tree(svo, scenes, case, seed)
        rays = torch.from_numpy(_pick_rays(tree.center(), case["n"], seed)).cuda()
        t = _march64(grid != 0, rays)
        return {"hit": None, "word": None, "t": t if case["n"] > 1 else t[0].cpu().numpy()}
    if kind == "view" and case["width"] * case["height"] <= 1 << 17:
        s = prepare(case, seed)
        occ = _grid(scenes, case["scene"], case["side"], seed) != 0
        return {"t": _march64(occ, s["rays"]), "word": None, "rgba8": None}
    return None
