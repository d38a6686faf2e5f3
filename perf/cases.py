"""The performance cases of this repository: what its users run, at the sizes they run it.

A case is a dict of plain values with a `kind`; `prepare` makes what a program holds before the
call (scene, plan, weights, input tensors), `run` makes one call through the public Python API of
vk_cinematic_gb300, `work` says what a pass cannot do without and `exact` gives the same outputs
in 64 bits from plain torch and numpy where that is feasible.

Kinds:
  frame       Renderer.frame: a whole image into a host buffer, as the offline renderer's caller
              takes it
  crop        SceneRenderer.render: a window with its G-buffers on the device, the denoiser's
              training and input renders
  preview     an animated scene: every object added again, the object BVH rebuilt, one frame, tone
              mapped to 8 bits on the device
  closest     Scene.intersect_closest_device: incoherent rays against a triangle soup
  query       Scene.intersect: a host batch of scene queries (editor picks, visibility probes)
  batch       Batch.launch: many scenes of uneven size in one launch
  compute     ComputePTScene.render_tiles: the compute-shader path tracer
  bake        create_cube_map and create_irradiance_cube_map: the application's environment bake
  denoise     KPCNN.denoise: the network on one frame
  train       KPCNN.train_step: forward, backward and Adam on a batch of crops
"""

from __future__ import annotations

import math

import numpy as np
import torch

from vk_cinematic_gb300 import denoiser, gbsp, scenes

_SHARED = {}


def _runtime():
    """The program's one runtime and its stream (torch work goes to the same stream)."""
    if not _SHARED:
        s = torch.cuda.Stream()
        _SHARED["stream"] = s
        _SHARED["rt"] = gbsp.Runtime(0, stream=s.cuda_stream)
    return _SHARED["rt"], _SHARED["stream"]


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # the smallest image anybody renders: the reference's own test scene, 128 x 128
        dict(name="frame_small", kind="frame", scene="sphere", width=128, height=128, spp=8,
             bounces=3, spheres=1, level=3, watertight=False),
        # the headline frame: 1080p, 64 samples, 5 bounces, 257 objects, 5.2 M triangles
        dict(name="frame_1080p", kind="frame", scene="spheres", width=1920, height=1080, spp=64,
             bounces=5, spheres=256, level=5, watertight=False),
        # an odd-sized product shot with closed meshes (watertight intersections, deeper paths)
        dict(name="frame_odd_watertight", kind="frame", scene="spheres", width=641, height=359,
             spp=7, bounces=8, spheres=61, level=4, watertight=True),
        # one training crop of the denoiser's dataset: 128 x 128, 4 samples, G-buffers
        dict(name="crop_gbuffer", kind="crop", width=1920, height=1080, side_x=128, side_y=128,
             spp=4, bounces=5, spheres=256, level=5),
        # interactive preview of an animated scene: 257 objects moved every frame, 1 sample
        dict(name="preview_animated", kind="preview", width=960, height=540, spp=1, bounces=3,
             spheres=256, level=4),
        # incoherent closest hits: 2^20 rays against a soup of 2^18 triangles
        dict(name="closest_soup", kind="closest", triangles=1 << 18, rays=1 << 20),
        # scene queries on a host batch of ragged size
        dict(name="query_host", kind="query", rays=20011, spheres=24, level=3),
        # twelve scenes of 1 k to 1 M triangles, 64^2 to 640^2 pixels, 1 to 64 samples
        dict(name="batch_uneven", kind="batch", count=12, max_side=640, max_spp=64,
             max_triangles=1000000, layout=4),
        # the compute-shader path tracer on a quarter-size window of its test scene
        dict(name="compute_tiles", kind="compute", width=512, height=384, spheres=16, level=3),
        # the application's environment bake: a 1024^2 cube map and a 32^2 irradiance map
        # (uniform grid) from a 2048 x 1024 image
        dict(name="bake_1024", kind="bake", eq_width=2048, eq_height=1024, size=1024, irr_size=32,
             random=False, spp=32),
        # the denoiser serving a 1080p frame
        dict(name="denoise_1080p", kind="denoise", width=1920, height=1080),
        # its training step on the usual batch, the backward direction
        dict(name="train_16x128", kind="train", batch=16, height=128, width=128),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "crop", "preview", "closest", "query", "batch", "compute",
                       "bake", "denoise", "train"])
    if kind == "frame":
        w, h = _log(rng, 64, 1920), _log(rng, 64, 1080)
        bounces = rng.randint(1, 8)
        # at most the path vertices of the headline frame
        spp = _log(rng, 1, max(1, min(64, int(1920 * 1080 * 64 * 5 / (w * h * bounces * 2)))))
        return dict(kind=kind, scene=rng.choice(["sphere", "spheres", "spheres"]), width=w,
                    height=h, spp=spp, bounces=bounces, spheres=_log(rng, 1, 256),
                    level=rng.randint(1, 5), watertight=rng.random() < 0.25)
    if kind == "crop":
        return dict(kind=kind, width=1920, height=1080, side_x=_log(rng, 32, 512),
                    side_y=_log(rng, 32, 512), spp=_log(rng, 1, 64), bounces=rng.randint(2, 6),
                    spheres=_log(rng, 16, 256), level=rng.randint(3, 5))
    if kind == "preview":
        return dict(kind=kind, width=_log(rng, 240, 1920), height=_log(rng, 135, 1080),
                    spp=rng.randint(1, 4), bounces=rng.randint(1, 4), spheres=_log(rng, 4, 512),
                    level=rng.randint(2, 5))
    if kind == "closest":
        return dict(kind=kind, triangles=_log(rng, 1000, 1 << 18), rays=_log(rng, 4096, 1 << 22))
    if kind == "query":
        return dict(kind=kind, rays=_log(rng, 100, 200000), spheres=_log(rng, 1, 64),
                    level=rng.randint(1, 3))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 16), max_side=_log(rng, 128, 640),
                    max_spp=_log(rng, 4, 64), max_triangles=_log(rng, 10000, 1000000),
                    layout=rng.randint(0, 1 << 20))
    if kind == "compute":
        return dict(kind=kind, width=_log(rng, 64, 640), height=_log(rng, 64, 480),
                    spheres=_log(rng, 1, 32), level=rng.randint(1, 3))
    if kind == "bake":
        h = _log(rng, 128, 1024)
        return dict(kind=kind, eq_width=2 * h, eq_height=h, size=_log(rng, 64, 1024),
                    irr_size=_log(rng, 8, 64), random=rng.random() < 0.5, spp=_log(rng, 8, 128))
    if kind == "denoise":
        return dict(kind=kind, width=_log(rng, 128, 1920), height=_log(rng, 128, 1080))
    return dict(kind="train", batch=rng.randint(1, 16), height=_log(rng, 48, 128),
                width=_log(rng, 48, 128))


# ---- inputs ---------------------------------------------------------------------------------

def _scene(case, seed):
    if case.get("scene") == "sphere":
        s = scenes.config1_scene(case["width"], case["height"], case["spp"], seed=seed)
        s.max_bounces = case["bounces"]
        return s
    return scenes.config3_scene(case["width"], case["height"], case["spp"], case["bounces"],
                                case["spheres"], case["level"], seed=seed)


def _batch_scenes(case, seed):
    """Config-4-style scenes whose sizes follow from the case and whose contents from the seed."""
    lay = np.random.default_rng(case["layout"])
    out = []
    for k in range(case["count"]):
        tris = math.exp(lay.uniform(math.log(1000), math.log(case["max_triangles"])))
        level = 5
        while level > 1 and 20 * 4 ** level > tris:
            level -= 1
        spheres = int(max(1, min(4096, round(tris / (20 * 4 ** level)))))
        side = int(round(math.exp(lay.uniform(math.log(64), math.log(case["max_side"])))))
        spp = int(round(math.exp(lay.uniform(0.0, math.log(case["max_spp"])))))
        out.append(scenes.config3_scene(side, side, spp, int(lay.integers(1, 9)), spheres, level,
                                        seed=seed * 1000 + k))
    return out


def _frame_inputs(shape, seed):
    """A noisy frame and its G-buffers with the statistics of a few-sample render: smooth shading
    under per-pixel noise with rare bright samples, piecewise constant albedo and normals, sky
    pixels without any."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    b, h, w = shape

    def smooth(c, cells):
        t = torch.rand((b, c, cells, cells), generator=g, device="cuda")
        return torch.nn.functional.interpolate(t, size=(h, w), mode="bilinear",
                                               align_corners=False).permute(0, 2, 3, 1)

    clean = smooth(3, 9) * 1.5
    noise = torch.empty((b, h, w, 1), device="cuda").log_normal_(-0.3, 0.7, generator=g)
    rad = torch.ones((b, h, w, 4), device="cuda")
    rad[..., :3] = torch.clamp(clean * noise, 0, 40)
    aov = torch.zeros((b, h, w, 8), device="cuda")
    aov[..., 0:3] = torch.round(smooth(3, 17) * 6) / 6
    aov[..., 3] = 2 + 20 * smooth(1, 7)[..., 0]
    n = smooth(3, 21) * 2 - 1
    aov[..., 4:7] = n / n.norm(dim=-1, keepdim=True).clamp_min(1e-3)
    aov[..., 7] = 1
    aov *= (smooth(1, 5) > 0.25).float()
    return rad.contiguous(), aov.contiguous(), clean.contiguous()


def prepare(case, seed):
    rt, stream = _runtime()
    kind = case["kind"]
    st = dict(case=case, seed=seed, stream=stream, rt=rt)
    with torch.cuda.stream(stream):
        if kind == "frame":
            s = _scene(case, seed)
            opt = gbsp.default_options(spp=case["spp"], max_bounces=case["bounces"], seed=seed)
            st["scene"], st["ms"], st["rend"] = gbsp.upload_scene(rt, s, opt)
            if case["watertight"]:
                st["scene"].set_intersection(gbsp.ISECT_WATERTIGHT)
            # the caller's image: page-locked, as a program that keeps one has it
            st["host"] = torch.zeros((case["height"], case["width"], 4)).pin_memory()
            st["pixels"] = st["host"].numpy()
        elif kind == "crop":
            st["sr"] = denoiser.SceneRenderer(rt, _scene(case, seed))
            r = np.random.default_rng(seed)
            st["x0"] = int(r.integers(0, case["width"] - case["side_x"]))
            st["y0"] = int(r.integers(0, case["height"] - case["side_y"]))
        elif kind == "preview":
            s = _scene(case, seed)
            opt = gbsp.default_options(spp=case["spp"], max_bounces=case["bounces"], seed=seed)
            st["scene"], st["ms"], st["rend"] = gbsp.upload_scene(rt, s, opt)
            st["objects"] = s.objects
        elif kind == "closest":
            s = scenes.config2_scene(case["triangles"], seed=seed)
            st["scene"], st["ms"], _ = gbsp.upload_scene(rt, s)
            rays = scenes.soup_rays(case["rays"], seed=seed + 1)
            packed = np.zeros((case["rays"], 8), np.float32)
            packed[:, 0:3], packed[:, 4:7] = rays[:, :3], rays[:, 3:]
            st["rays"] = torch.from_numpy(packed).cuda()
        elif kind == "query":
            st["desc"], st["rays"] = _query_inputs(case, seed)
            st["scene"], st["ms"], _ = gbsp.upload_scene(rt, st["desc"])
        elif kind == "batch":
            st["parts"] = [gbsp.upload_scene(rt, s) for s in _batch_scenes(case, seed)]
            rends = [p[2] for p in st["parts"]]
            st["images"] = [torch.zeros((r.height, r.width, 4), device="cuda") for r in rends]
            st["batch"] = gbsp.Batch(rt, rends, [i.data_ptr() for i in st["images"]])
        elif kind == "compute":
            s = scenes.compute_pt_scene(case["spheres"], case["level"], seed=seed)
            # the shader's RNG is seeded by tile index alone: the camera is what a new call moves
            cam = s["camera_transform"].copy()
            cam[12:15] += np.random.default_rng(seed).uniform(-2, 2, 3).astype(np.float32)
            st["scene"] = gbsp.ComputePTScene(rt, s["vertices"], s["indices"], s["meshes"],
                                              s["model"], s["inv_model"], s["entities"],
                                              s["texture"])
            st["view"] = gbsp.cpt_view(case["width"], case["height"], camera_transform=cam)
            st["tiles"] = np.arange((case["width"] // 16) * (case["height"] // 16),
                                    dtype=np.uint32)
        elif kind == "bake":
            st["eq"] = torch.from_numpy(scenes.equirect_hdri(case["eq_width"], case["eq_height"],
                                                             seed)).cuda()
        elif kind == "denoise":
            st["net"] = denoiser.KPCNN(seed=seed)
            st["rad"], st["aov"], _ = _frame_inputs((1, case["height"], case["width"]), seed)
        elif kind == "train":
            st["net"] = denoiser.KPCNN(seed=seed)
            st["rad"], aov, clean = _frame_inputs((case["batch"], case["height"], case["width"]),
                                                  seed)
            st["feats"] = st["net"].features(st["rad"], aov)
            st["target"] = torch.ones_like(st["rad"])
            st["target"][..., :3] = clean
    return st


def _query_inputs(case, seed):
    s = scenes.config3_scene(0, 0, 1, 1, case["spheres"], case["level"], seed=seed)
    r = np.random.default_rng(seed + 1)
    o = r.uniform([-10, 0.5, -10], [10, 8, 10], (case["rays"], 3)).astype(np.float32)
    d = r.standard_normal((case["rays"], 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return s, np.concatenate([o, d], axis=1)


# ---- one pass -------------------------------------------------------------------------------

def run(st):
    case, kind, stream = st["case"], st["case"]["kind"], st["stream"]
    with torch.cuda.stream(stream):
        if kind == "frame":
            st["rend"].frame(pixels=st["pixels"])
            return st["host"]
        if kind == "crop":
            rad, aov = st["sr"].render(st["x0"], st["y0"], case["side_x"], case["side_y"],
                                       case["spp"], st["seed"], aov=True)
            return [rad, aov]
        if kind == "preview":
            scene, rend = st["scene"], st["rend"]
            scene.clear_objects()
            for o in st["objects"]:
                scene.add_object(o.mesh, o.material, o.position, o.rotation, o.scale)
            scene.build_broadphase()
            rend.frame_async()
            frame = torch.empty((case["height"], case["width"], 4), device="cuda")
            rend.copy_region(0, 0, case["width"], case["height"], frame.data_ptr())
            return [frame, gbsp.tonemap(frame, stream=stream.cuda_stream)]
        if kind == "closest":
            n = case["rays"]
            t = torch.empty(n, device="cuda")
            tri = torch.empty(n, dtype=torch.int32, device="cuda")
            obj = torch.empty(n, dtype=torch.int32, device="cuda")
            st["scene"].intersect_closest_device(n, st["rays"].data_ptr(), t.data_ptr(),
                                                 tri.data_ptr(), obj.data_ptr())
            return [t, tri, obj]
        if kind == "query":
            hits, mats, _ = st["scene"].intersect(st["rays"])
            return [hits, mats.view(np.int32)]
        if kind == "batch":
            st["batch"].launch(metrics=False)
            return st["images"]
        if kind == "compute":
            img = torch.zeros((case["height"], case["width"], 4), device="cuda")
            st["scene"].render_tiles(st["view"], st["tiles"], img.data_ptr(), metrics=False)
            return img
        if kind == "bake":
            mode = gbsp.IRRADIANCE_RANDOM if case["random"] else gbsp.IRRADIANCE_UNIFORM
            sid = stream.cuda_stream
            return [gbsp.create_cube_map(st["eq"], case["size"], case["size"], stream=sid),
                    gbsp.create_irradiance_cube_map(st["eq"], case["irr_size"], case["irr_size"],
                                                    case["spp"], mode, stream=sid)]
        if kind == "denoise":
            return st["net"].denoise(st["rad"], st["aov"])
        net = st["net"]
        loss = net.train_step(st["feats"], st["rad"], st["target"])
        return dict(loss=loss, w=net.w, b=net.b, m=[x[0] for x in net.state],
                    mb=[x[2] for x in net.state])


# ---- what a pass cannot do without ----------------------------------------------------------

# rays per path of the open scenes here (about half of the bounce rays leave), flops of walking
# one ray: two box tests per level of a balanced tree over the triangles and one triangle test
def _ray_flops(triangles):
    return 2 * 17 * max(1.0, math.log2(max(2, triangles))) + 50


def _trace_work(paths, bounces, pixels, mesh_tris, objects):
    rays = paths * min(bounces, 2)
    return {"bytes": pixels * 16 + mesh_tris * 48 + objects * 96,
            "flops": rays * (_ray_flops(mesh_tris) + _ray_flops(objects)) + paths * 150}


def work(case):
    kind = case["kind"]
    if kind in ("frame", "crop", "preview"):
        if kind == "crop":
            pixels = case["side_x"] * case["side_y"]
        else:
            pixels = case["width"] * case["height"]
        w = _trace_work(pixels * case["spp"], case["bounces"], pixels, 20 * 4 ** case["level"],
                        case["spheres"] + 1)
        if kind == "crop":
            w["bytes"] += pixels * 32
        if kind == "preview":
            w["bytes"] += pixels * 4
        return w
    if kind == "closest":
        n = case["rays"]
        return {"bytes": n * (32 + 12) + case["triangles"] * 48,
                "flops": n * _ray_flops(case["triangles"])}
    if kind == "query":
        n, tris = case["rays"], 20 * 4 ** case["level"]
        return {"bytes": n * (24 + 28) + tris * 48, "flops": n * 2 * _ray_flops(tris)}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        lay = np.random.default_rng(case["layout"])
        for _ in range(case["count"]):
            tris = math.exp(lay.uniform(math.log(1000), math.log(case["max_triangles"])))
            side = int(round(math.exp(lay.uniform(math.log(64), math.log(case["max_side"])))))
            spp = int(round(math.exp(lay.uniform(0.0, math.log(case["max_spp"])))))
            w = _trace_work(side * side * spp, int(lay.integers(1, 9)), side * side,
                            min(tris, 20480), max(1, tris / 20480))
            total = {k: total[k] + w[k] for k in total}
        return {k: int(v) for k, v in total.items()}
    if kind == "compute":
        pixels = (case["width"] // 16) * (case["height"] // 16) * 256
        tris = 20 * 4 ** case["level"]
        # every ray meets every entity; a tree over each entity's triangles would do for the rest
        return {"bytes": pixels * 16 + tris * 36,
                "flops": pixels * 2 * (case["spheres"] + 3) * _ray_flops(tris)}
    if kind == "bake":
        texels, irr = 6 * case["size"] ** 2, 6 * case["irr_size"] ** 2
        samples = irr * (case["spp"] if case["random"] else 1008)
        return {"bytes": (texels + irr + case["eq_width"] * case["eq_height"]) * 16,
                "flops": (texels + samples) * 100}
    macs = sum(9 * cin * cout for cin, cout, _ in denoiser.LAYERS)
    if kind == "denoise":
        pixels = case["width"] * case["height"]
        return {"bytes": pixels * (16 + 32 + 16), "flops": pixels * (2 * macs + 200)}
    pixels = case["batch"] * case["height"] * case["width"]
    params = sum(9 * cin * cout + cout for cin, cout, _ in denoiser.LAYERS)
    return {"bytes": pixels * (32 + 16 + 16) + params * (12 + 12 + 2),
            "flops": pixels * (3 * 2 * macs - 2 * 9 * 16 * 48 + 400)}


# ---- the same outputs in 64 bits ------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "query":
        return _exact_query(case, seed)
    if kind == "bake":
        return _exact_bake(case, seed)
    if kind == "denoise":
        return _exact_denoise(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    # paths are chaotic: a rounding at one bounce sends the next ray elsewhere, so a 64-bit
    # render is another sample of the same image; soups of 2^18 triangles take too long to
    # brute-force
    return None


def _rot(q):
    x, y, z, w = (float(v) for v in q)
    return np.array([[1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * z * w, 2 * x * z + 2 * y * w],
                     [2 * x * y + 2 * z * w, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * x * w],
                     [2 * x * z - 2 * y * w, 2 * y * z + 2 * x * w, 1 - 2 * x * x - 2 * y * y]])


def _exact_query(case, seed):
    """Brute-force Moller-Trumbore over every triangle of every object."""
    s, rays = _query_inputs(case, seed)
    dev = "cuda"
    o = torch.from_numpy(rays[:, :3]).double().to(dev)
    d = torch.from_numpy(rays[:, 3:]).double().to(dev)
    n = len(rays)
    best = torch.full((n,), math.inf, dtype=torch.float64, device=dev)
    out = torch.zeros((n, 6), dtype=torch.float64, device=dev)
    out[:, 0] = -1
    for ob in s.objects:
        v, idx, _ = s.meshes[ob.mesh]
        rot = torch.from_numpy(_rot(ob.rotation)).to(dev)
        scale = torch.from_numpy(ob.scale.astype(np.float64)).to(dev)
        pos = torch.from_numpy(ob.position.astype(np.float64)).to(dev)
        tri = torch.from_numpy(v[idx.astype(np.int64)].reshape(-1, 3, 8)).double().to(dev)
        p = (tri[..., :3] * scale) @ rot.T + pos
        a, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        nl = torch.linalg.cross(tri[:, 1, :3] - tri[:, 0, :3], tri[:, 2, :3] - tri[:, 0, :3])
        nrm = (nl * scale) @ rot.T
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        step = max(1, (1 << 24) // len(tri))
        for k in range(0, n, step):
            dd, oo = d[k:k + step, None], o[k:k + step, None]
            pv = torch.linalg.cross(dd.expand(-1, len(tri), -1), e2[None].expand(dd.shape[0], -1, -1))
            tv = oo - a[None]
            qv = torch.linalg.cross(tv, e1[None].expand(dd.shape[0], -1, -1))
            inv = 1.0 / (pv * e1[None]).sum(-1)
            t = (qv * e2[None]).sum(-1) * inv
            u = (pv * tv).sum(-1) * inv
            w = (qv * dd).sum(-1) * inv
            front = (dd[:, 0] @ torch.linalg.cross(e1, e2).T) < 0
            hit = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & front
            tt, j = torch.where(hit, t, torch.full_like(t, math.inf)).min(dim=1)
            near = tt < best[k:k + step]
            rows = torch.nonzero(near)[:, 0]
            jj = j[rows]
            uu, ww = u[rows, jj], w[rows, jj]
            uv = tri[jj, 0, 6:8] * (1 - uu - ww)[:, None] + tri[jj, 1, 6:8] * uu[:, None] + \
                tri[jj, 2, 6:8] * ww[:, None]
            out[k + rows] = torch.cat([tt[rows, None], nrm[jj], uv], dim=1)
            best[k + rows] = tt[rows]
    return [out, None]


def _face_directions(size):
    basis = [((1, 0, 0), (0, 1, 0), (0, 0, -1)), ((-1, 0, 0), (0, 1, 0), (0, 0, 1)),
             ((0, 1, 0), (0, 0, -1), (1, 0, 0)), ((0, -1, 0), (0, 0, 1), (1, 0, 0)),
             ((0, 0, 1), (0, 1, 0), (1, 0, 0)), ((0, 0, -1), (0, 1, 0), (-1, 0, 0))]
    b = torch.tensor(basis, dtype=torch.float64, device="cuda")
    c = torch.arange(size, dtype=torch.float64, device="cuda") / size
    fx = (c * 2 - 1)[None, None, :, None]
    fy = ((1 - c) * 2 - 1)[None, :, None, None]
    d = b[:, 0][:, None, None] + b[:, 2][:, None, None] * fx + b[:, 1][:, None, None] * fy
    return d / d.norm(dim=-1, keepdim=True), b[:, 1]


def _sample(eq, d):
    """Bilinear, clamped equirectangular lookup along directions d (..., 3)."""
    h, w, _ = eq.shape
    inc = torch.atan2(torch.sqrt(d[..., 0] ** 2 + d[..., 2] ** 2), d[..., 1])
    az = torch.atan2(d[..., 2], d[..., 0])
    az = torch.where(az < 0, az + 2 * math.pi, az)
    px = torch.clamp(az / (2 * math.pi) * w - 0.5, min=0)
    py = torch.clamp((1 - (torch.cos(inc) * 0.5 + 0.5)) * h - 0.5, min=0)
    x0, y0 = px.floor(), py.floor()
    fx, fy = (px - x0)[..., None], (py - y0)[..., None]
    xa, ya = x0.long().clamp(max=w - 1), y0.long().clamp(max=h - 1)
    xb, yb = (x0.long() + 1).clamp(max=w - 1), (y0.long() + 1).clamp(max=h - 1)
    top = eq[ya, xa] * (1 - fx) + eq[ya, xb] * fx
    bot = eq[yb, xa] * (1 - fx) + eq[yb, xb] * fx
    return top * (1 - fy) + bot * fy


def _exact_bake(case, seed):
    eq = torch.from_numpy(scenes.equirect_hdri(case["eq_width"], case["eq_height"],
                                               seed)).cuda().double()
    return [_sample(eq, _face_directions(case["size"])[0]), _exact_irradiance(case, eq)]


def _exact_irradiance(case, eq):
    size = case["irr_size"]
    n, up = _face_directions(size)
    out = torch.ones((6, size, size, 4), dtype=torch.float64, device="cuda")
    if case["random"]:
        total = 6 * size * size * case["spp"] * 3
        r = np.empty(total)
        s = 0x45BA12F3
        for k in range(total):
            s ^= (s << 13) & 0xFFFFFFFF
            s ^= s >> 17
            s ^= (s << 5) & 0xFFFFFFFF
            r[k] = s >> 1
        r = torch.from_numpy(-1 + 2 * (r / 0x7FFFFFFF)).cuda().reshape(6, size, size, case["spp"], 3)
        d = n[..., None, :] + r.flip(-1)
        d = d / d.norm(dim=-1, keepdim=True)
        cosine = (d * n[..., None, :]).sum(-1, keepdim=True)
        d, cosine = torch.where(cosine < 0, -d, d), cosine.abs()
        for f in range(6):
            out[f, ..., :3] = torch.clamp(_sample(eq, d[f])[..., :3] * cosine[f], 0, 10).mean(-2)
        return out
    grid = []
    phi, step = np.float32(0), np.float32(0.1)
    pi = np.float32(3.14159265359)
    while phi < np.float32(2) * pi:
        theta = np.float32(0)
        while theta < np.float32(0.5) * pi:
            grid.append((float(phi), float(theta)))
            theta += step
        phi += step
    g = torch.tensor(grid, dtype=torch.float64, device="cuda")
    st, ct = torch.sin(g[:, 1]), torch.cos(g[:, 1])
    lx, lz = st * torch.cos(g[:, 0]), st * torch.sin(g[:, 0])
    for f in range(6):
        nn = n[f].reshape(-1, 1, 3)
        t = torch.linalg.cross(up[f].expand(nn.shape[0], 1, 3), nn)
        t = t / t.norm(dim=-1, keepdim=True)
        b = torch.linalg.cross(nn, t)
        b = b / b.norm(dim=-1, keepdim=True)
        d = nn * ct[None, :, None] + t * lx[None, :, None] + b * lz[None, :, None]
        rad = torch.clamp(_sample(eq, d)[..., :3], 0, 10) * (ct * st)[None, :, None]
        out[f, ..., :3] = (math.pi * rad.mean(1)).reshape(size, size, 3)
    return out


def _conv(x, w, b):
    """3 x 3 convolution with zero padding: x (B, H, W, Cin), w (9, Cout, Cin)."""
    _, h, wd, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = b.expand(x.shape[0], h, wd, -1)
    for tap in range(9):
        y = y + p[:, tap // 3:tap // 3 + h, tap % 3:tap % 3 + wd] @ w[tap].T
    return y


def _features64(rad, aov):
    f = torch.zeros(rad.shape[:3] + (16,), dtype=torch.float64, device="cuda")
    f[..., 0:3] = torch.log1p(rad[..., :3].double().clamp_min(0))
    f[..., 3:6], f[..., 6:9] = aov[..., 0:3].double(), aov[..., 4:7].double()
    d = aov[..., 3].double().clamp_min(0)
    f[..., 9] = d / (1 + d)
    return f


def _filter64(logits, rad):
    w = torch.softmax(logits[..., :25], dim=-1)
    _, h, wd, _ = rad.shape
    p = torch.nn.functional.pad(rad[..., :3].double().permute(0, 3, 1, 2), (2, 2, 2, 2),
                                mode="replicate").permute(0, 2, 3, 1)
    return sum(w[..., k:k + 1] * p[:, k // 5:k // 5 + h, k % 5:k % 5 + wd] for k in range(25))


def _network64(x, ws, bs):
    last = len(ws) - 1
    for li, (w, b) in enumerate(zip(ws, bs)):
        x = _conv(x, w, b)
        if li < last:
            x = torch.relu(x)
    return x


def _weights64(seed):
    """The network's initial weights: scaled normals from torch's CPU generator, as BF16."""
    g = torch.Generator().manual_seed(seed)
    out = []
    for cin, cout, epi in denoiser.LAYERS:
        fan = 9 * (denoiser.N_FEATURES if cin == denoiser.FEATURE_CHANNELS else cin)
        w = torch.randn((9, cout, cin), generator=g) * (math.sqrt(2.0 / fan) *
                                                        (0.1 if epi == 1 else 1.0))
        if cin == denoiser.FEATURE_CHANNELS:
            w[:, :, denoiser.N_FEATURES:] = 0
        if epi == 1:
            w[:, 25:, :] = 0
        out.append(w.cuda())
    return out


def _exact_denoise(case, seed):
    rad, aov, _ = _frame_inputs((1, case["height"], case["width"]), seed)
    ws = [w.to(torch.bfloat16).double() for w in _weights64(seed)]
    bs = [torch.zeros(w.shape[1], dtype=torch.float64, device="cuda") for w in ws]
    out = torch.ones(rad.shape, dtype=torch.float64, device="cuda")
    out[..., :3] = _filter64(_network64(_features64(rad, aov), ws, bs), rad)
    return out


def _exact_train(case, seed):
    rad, aov, clean = _frame_inputs((case["batch"], case["height"], case["width"]), seed)
    master = _weights64(seed)
    ws = [w.to(torch.bfloat16).double().requires_grad_() for w in master]
    bs = [torch.zeros(w.shape[1], dtype=torch.float64, device="cuda").requires_grad_() for w in ws]
    o = _filter64(_network64(_features64(rad, aov).to(torch.bfloat16).double(), ws, bs), rad)
    r = clean.double()
    loss = ((o - r) ** 2 / (r * r + 0.01)).mean()
    loss.backward()

    def adam(p, g):
        return p - 1e-4 * g / (g.abs() + 1e-8)

    return dict(loss=loss.detach().reshape(1),
                w=[adam(p.double(), w.grad) for p, w in zip(master, ws)],
                # biases start at 0 and move by lr * sign(gradient): no relative error to speak of
                b=[None] * len(bs),
                m=[0.1 * w.grad for w in ws], mb=[0.1 * b.grad for b in bs])
