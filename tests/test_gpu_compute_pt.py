"""The compute-shader path tracer on the GPU (gbsp_cpt_*) against its CPU
restatement: every operation is a basic IEEE operation or sqrt, so images
and counters must agree bit for bit."""

import numpy as np
import pytest

from oracle import pyoracle
from vk_cinematic_gb300 import gbsp, scenes

pytestmark = pytest.mark.gpu


def render_gpu(s, width, height, tiles, fill=0.0):
    import torch

    rt = gbsp.Runtime()
    sc = gbsp.ComputePTScene(rt, s["vertices"], s["indices"], s["meshes"], s["model"],
                             s["inv_model"], s["entities"], s.get("texture"))
    img = torch.full((height, width, 4), fill, dtype=torch.float32, device="cuda")
    view = gbsp.cpt_view(width, height, 16, 0.8, s["camera_transform"])
    m = sc.render_tiles(view, tiles, img.data_ptr())
    out = img.cpu().numpy()
    sc.close()
    return out, m.as_dict()


@pytest.mark.parametrize("level,n_spheres", [(1, 16), (2, 24)])
def test_full_image_bit_exact(gpu_lib, level, n_spheres):
    pyoracle.build_port()
    s = scenes.compute_pt_scene(n_spheres=n_spheres, level=level)
    w, h = 256, 192
    tiles = np.arange((w // 16) * (h // 16))
    ref, c = pyoracle.compute_pt_tiles(s, w, h, 16, 0.8, tiles)
    got, m = render_gpu(s, w, h, tiles)
    same = got.view(np.uint32) == ref.view(np.uint32)
    assert same.all(), f"{(~same).sum()} words differ; first at {np.argwhere(~same)[:3]}"
    assert m["rays_traced"] == int(c[0])
    assert m["ray_hit_count"] == int(c[1])
    assert m["triangle_tests"] == int(c[2])
    assert (ref[..., :3] > 0).mean() > 0.05  # the light is seen


def test_tile_subset_and_ragged_image(gpu_lib):
    pyoracle.build_port()
    s = scenes.compute_pt_scene(n_spheres=5, level=3)
    w, h = 200, 120  # tiles clipped at the right and bottom edges
    tiles = np.array([0, 11, 12, 35, 40, 77, 3])  # 77 lies outside the image: no pixels
    ref = np.full((h, w, 4), -3.0, np.float32)
    ref, c = pyoracle.compute_pt_tiles(s, w, h, 16, 0.8, tiles, image=ref)
    got, m = render_gpu(s, w, h, tiles, fill=-3.0)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert m["rays_traced"] == int(c[0])


def test_rejects_bad_input(gpu_lib):
    s = scenes.compute_pt_scene(n_spheres=1, level=0)
    rt = gbsp.Runtime()
    bad = s["entities"].copy()
    bad[0, 0] = 9  # no mesh 9
    with pytest.raises(gbsp.GbspError, match="out of range"):
        gbsp.ComputePTScene(rt, s["vertices"], s["indices"], s["meshes"], s["model"],
                            s["inv_model"], bad, s["texture"])
    idx = s["indices"].copy()
    idx[0] = 10 ** 6
    with pytest.raises(gbsp.GbspError, match="vertex index"):
        gbsp.ComputePTScene(rt, s["vertices"], idx, s["meshes"], s["model"], s["inv_model"],
                            s["entities"], s["texture"])


def soup_mesh(rng, n, sliver):
    """n triangles around the origin, a share of them slivers, some without area."""
    p = rng.uniform(-1.5, 1.5, (n, 1, 3)) + rng.uniform(-0.6, 0.6, (n, 3, 3))
    thin = rng.random(n) < sliver
    p[thin, 2] = p[thin, 0] + (p[thin, 1] - p[thin, 0]) * rng.random((thin.sum(), 1)) + \
        rng.uniform(-1e-5, 1e-5, (thin.sum(), 3))
    flat = rng.random(n) < sliver / 4
    p[flat, 2] = p[flat, 1]
    v = np.zeros((3 * n, 8), np.float32)
    v[:, 0:3] = p.reshape(-1, 3)
    v[:, 6:8] = rng.random((3 * n, 2))
    return v, np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("entities,tris,sliver", [(0, 5, 0.0), (1, 1, 0.0), (1, 17, 0.3),
                                                  (33, 16, 0.1), (70, 3, 0.0), (2, 700, 0.3),
                                                  (3, 2100, 0.0), (12, 400, 1.0)])
def test_clusters_lose_no_hit(gpu_lib, entities, tris, sliver):
    """Triangle clusters against the oracle's brute force, bit for bit: cluster
    and warp-step remainders (1, 16, 17 triangles; more entities than a warp
    has lanes; lists that are run in several parts), meshes without triangles,
    slivers and degenerate triangles, rotated, scaled and mirrored entities."""
    pyoracle.build_port()
    rng = np.random.default_rng(100 * entities + tris)
    sv, si = soup_mesh(rng, tris, sliver)
    pv, pi = scenes.plane()
    s = scenes.compute_pt_scene(n_spheres=1, level=0)
    s["vertices"] = np.concatenate([pv, sv]).astype(np.float32)
    s["indices"] = np.concatenate([pi, si]).astype(np.uint32)
    s["meshes"] = np.array([[len(pi), 0, 0], [len(si), len(pi), len(pv)], [0, 0, 0]], np.uint32)
    model, inv, ents = [], [], []
    for k in range(entities):
        m, i = scenes._trs(rng.uniform([-8, 0, -8], [8, 6, 8]), rng.uniform(-3, 3),
                           rng.uniform(0.3, 2.0, 3) * rng.choice([-1.0, 1.0], 3))
        model.append(m)
        inv.append(i)
        # a ground quad, an empty mesh now and then, the soup otherwise
        ents.append((0 if k == 1 else 2 if k % 9 == 5 else 1, [0, 2, 5][k % 3], k))
    s["model"] = np.array(model, np.float32).reshape(-1, 16)
    s["inv_model"] = np.array(inv, np.float32).reshape(-1, 16)
    s["entities"] = np.array(ents, np.uint32).reshape(-1, 3)
    s["texture"] = np.ascontiguousarray(rng.random((7, 13, 4)).astype(np.float32))
    w, h = 45, 37
    tiles = np.arange((w // 16) * 3)
    ref = np.zeros((h, w, 4), np.float32)
    ref, c = pyoracle.compute_pt_tiles(s, w, h, 16, 0.8, tiles, image=ref)
    got, m = render_gpu(s, w, h, tiles)
    same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), f"{(~same).sum()} words differ"
    assert (m["rays_traced"], m["ray_hit_count"], m["triangle_tests"]) == tuple(int(v) for v in c[:3])


@pytest.mark.parametrize("scale", [1e19, 1e22, 2e22])
def test_huge_entities_lose_no_hit(gpu_lib, scale):
    """Entities scaled until the squares of an object-space direction are
    denormal, so that its normalisation no longer gives unit length: the image
    is the brute-force oracle's, bit for bit."""
    pyoracle.build_port()
    s = scenes.compute_pt_scene(n_spheres=1, level=0)
    v, i = gbsp.icosphere(3)[:2]
    s["vertices"], s["indices"] = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(i, np.uint32)
    s["meshes"] = np.array([[len(i), 0, 0]], np.uint32)
    model, inv, ents = [], [], []
    for x in (-1, 0, 1):
        for y in (-1, 0, 1):
            for z in (-1, 0, 1):
                if (x, y, z) == (0, 0, 0):
                    continue
                m, n = scenes._trs(np.array([x, y, z]) * 3.0 * scale, 1.0, np.full(3, scale))
                ents.append((0, [5, 0][len(ents) % 2], len(ents)))
                model.append(m)
                inv.append(n)
    s["model"] = np.array(model, np.float32).reshape(-1, 16)
    s["inv_model"] = np.array(inv, np.float32).reshape(-1, 16)
    s["entities"] = np.array(ents, np.uint32)
    w, h = 48, 32
    tiles = np.arange(6)
    ref, c = pyoracle.compute_pt_tiles(s, w, h, 16, 0.8, tiles)
    got, m = render_gpu(s, w, h, tiles)
    same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), f"{(~same).sum()} words differ"
    assert (m["rays_traced"], m["ray_hit_count"]) == (int(c[0]), int(c[1]))
    assert m["ray_hit_count"] > 0
