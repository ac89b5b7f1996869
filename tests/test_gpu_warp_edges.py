"""GPU test of calls whose rays or pixels do not fill whole warps.

The traversal walks a warp's rays together, lanes without a ray following along, so the results
of a small or ragged call must equal those of the same rays and pixels inside a larger one, bit
for bit: ray sets around the warp (32) and block (128) sizes, and crops smaller than an 8x4 tile.
"""
import numpy as np
import pytest

import luminara_b200 as L
from luminara_b200 import workloads as W

from .helpers import random_rays, to_gpu_rays, to_orc_rays

pytestmark = pytest.mark.gpu

SCENES = {"box_room": (lambda: W.box_room(64, 48, 4), (0, 0, 0), (555, 555, 555)),
          "zoo": (lambda: W.material_zoo(64, 48, 4), (-6, 0, -4), (6, 8, 6)),
          "mesh": (lambda: W.dense_mesh(64, 48, 4, level=3), (-2, -1, -2), (2, 2, 2))}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_ragged_ray_sets_equal_the_whole_set(name):
    build, lo, hi = SCENES[name]
    sc = L.GpuScene(build()[0])
    rays = to_gpu_rays(*random_rays(np.random.default_rng(3), 4097, lo, hi))
    hits, occ = sc.intersect(rays), sc.occluded(rays)
    assert 0 < occ.sum()
    np.testing.assert_array_equal(occ != 0, hits["prim_id"] >= 0)
    for n in (1, 31, 32, 33, 127, 128, 129, 1000):
        assert sc.intersect(rays[:n]).tobytes() == hits[:n].tobytes(), n
        np.testing.assert_array_equal(sc.occluded(rays[:n]), occ[:n])
    sc.close()


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("crop", [(0, 0, 1, 1), (7, 3, 9, 5), (5, 6, 8, 4), (40, 30, 24, 18)])
def test_ragged_crops_equal_the_frame(name, crop):
    world, cfg = SCENES[name][0]()
    sc = L.GpuScene(world)
    frame, _ = sc.render(cfg)
    cfg.crop = crop
    part, _ = sc.render(cfg)
    x, y, w, h = crop
    np.testing.assert_array_equal(part, frame[y:y + h, x:x + w])
    sc.close()


def test_small_frames_and_strata_match_the_keyed_oracle():
    """Widths, heights and stratum counts around the tile (8x4) and the divisions of a path start."""
    import oracle as O
    close = total = 0
    for w, h in [(2, 2), (3, 5), (8, 4), (17, 9), (33, 2)]:
        for spp in (1, 3, 16, 30):
            world, cfg = W.box_room(w, h, spp, seed=100 * w + spp)
            sc = L.GpuScene(world)
            img, _ = sc.render(cfg)
            sc.close()
            ref = O.OracleScene(world).render(cfg, mode=O.MODE_KEYED)[0]
            near = (np.abs(img - ref) <= 2e-3 * (1 + np.abs(ref))).all(-1)   # the keyed renders' rule
            close, total = close + int(near.sum()), total + near.size
    assert close >= 0.97 * total, (close, total)


@pytest.mark.parametrize("name", ["box_room", "zoo", "spheres"])
@pytest.mark.parametrize("size", [(2, 2), (37, 21), (64, 48)])
def test_adaptive_classes_match_the_keyed_oracle(name, size):
    """The quad, other-materials and sphere builds of the adaptive kernel at ragged sizes and a last
    round of 9 strata (25 in all), none stopped (threshold 0), by the keyed renders' rule."""
    import oracle as O
    build = W.random_spheres if name == "spheres" else SCENES[name][0]
    world, cfg = build(*size, 20) if name == "spheres" else build()
    cfg.width, cfg.height, cfg.samples_per_pixel = size[0], size[1], 20
    cfg.adaptive, cfg.adaptive_threshold = True, 0.0
    sc = L.GpuScene(world)
    img, st = sc.render(cfg)
    sc.close()
    assert st.paths == 25 * size[0] * size[1]
    ref = O.OracleScene(world).render(cfg, mode=O.MODE_KEYED)[0]
    assert (np.abs(img - ref) <= 2e-3 * (1 + np.abs(ref))).all(-1).mean() >= (0.95 if name == "zoo" else 0.97)


@pytest.mark.parametrize("n_big,n_small", [(1, 0), (1, 40), (4, 40), (5, 40), (3, 0)])
def test_big_spheres_beside_the_tree(n_big, n_small):
    """Spheres of radius 32 and more stay out of a sphere scene's tree, up to four of them: every
    render mode gives the same image, and closest hits and occlusion are the oracle's."""
    import oracle as O
    from luminara_b200 import abi
    rng = np.random.default_rng(10 * n_big + n_small)
    w = L.World()
    for k in range(n_big):
        r = 32.0 if k == 1 else 100.0 * (k + 1)
        w.add(L.Sphere((40.0 * k, -r - 0.01 * k, 5.0 * k), r, L.Lambertian((0.3 + 0.1 * k, 0.5, 0.4))))
    for _ in range(n_small):
        w.add(L.Sphere(tuple(rng.uniform((-4, 0.2, -4), (4, 1.5, 4))), 0.3, L.Metal((0.8, 0.7, 0.6), 0.2)))
    w.camera = L.CameraConfig(look_from=(6, 2, 6), look_at=(0, 0.5, 0), aspect_ratio=37 / 21)
    cfg = L.RenderConfig(width=37, height=21, samples_per_pixel=9, max_depth=6, seed=5)
    sc = L.GpuScene(w)
    img, _ = sc.render(cfg)
    for mode in (abi.BATCH_WAVEFRONT, abi.BATCH_MEGAKERNEL, abi.BATCH_STREAMS):
        batch = L.Batch([sc], [cfg], config={"mode": mode})
        np.testing.assert_array_equal(batch.render()[0][0], img)
        batch.close()
    orc = O.OracleScene(w)
    for c in (cfg, L.RenderConfig(**{**cfg.__dict__, "background": abi.BG_STARFIELD, "bg_star_density": 0.2,
                                     "bg_star_brightness": 1.0})):
        got, ref = sc.render(c)[0], orc.render(c, mode=O.MODE_KEYED)[0]
        assert (np.abs(got - ref) <= 2e-3 * (1 + np.abs(ref))).all(-1).mean() >= 0.97
    o, d, t0, t1 = random_rays(rng, 2000, (-8, 0.05, -8), (8, 6, 8))
    hits, want = sc.intersect(to_gpu_rays(o, d, t0, t1)), orc.intersect(to_orc_rays(o, d, t0, t1))
    same = hits["prim_id"] == want["prim_id"]
    assert same.mean() >= 0.995 and (want["prim_id"] >= 0).any()
    hit = same & (want["prim_id"] >= 0)
    np.testing.assert_allclose(hits["t"][hit], want["t"][hit], rtol=2e-3, atol=2e-4)
    assert ((sc.occluded(to_gpu_rays(o, d, t0, t1)) != 0) == (want["prim_id"] >= 0)).mean() >= 0.995
    sc.close()


@pytest.mark.parametrize("kind,n", [("general", 16000), ("general", 17000), ("mesh", 6)])
def test_large_scene_builds_equal_the_other_modes(kind, n):
    """Scenes on both sides of the sizes from which warps turn to their leaves early: the same image in
    every render mode (the batch's kernels never do), and again."""
    from luminara_b200 import abi
    if kind == "mesh":
        world, cfg = W.dense_mesh(61, 35, 4, level=n)                      # 81,920 triangles
    else:
        world, cfg = W.uneven_scene(np.random.default_rng(n), n, 61, 35, 4)
    sc = L.GpuScene(world)
    img, _ = sc.render(cfg)
    for mode in (abi.BATCH_WAVEFRONT, abi.BATCH_MEGAKERNEL, abi.BATCH_STREAMS):
        batch = L.Batch([sc], [cfg], config={"mode": mode})
        np.testing.assert_array_equal(batch.render()[0][0], img)
        batch.close()
    np.testing.assert_array_equal(sc.render(cfg)[0], img)
    sc.close()


@pytest.mark.parametrize("size", [(64, 48), (128, 128), (320, 180), (640, 360)])
def test_task_plans_add_up_to_the_same_frame(size):
    """Frames whose plans split strata into groups of 1, 2, 4 and more: two stratum ranges, each with its
    own plan, add up to the whole frame's raw sums."""
    import torch
    world, cfg = W.box_room(*size, 16, max_depth=3)
    sc = L.GpuScene(world)
    def sums(begin, count):
        cfg.sample_begin, cfg.sample_count = begin, count
        t = torch.empty((size[1], size[0], 4), dtype=torch.int64, device="cuda")
        sc.render_sums_device(cfg, t.data_ptr())
        return t
    whole, parts = sums(0, 16), sums(0, 5) + sums(5, 11)
    assert torch.equal(whole, parts)
    cfg.sample_begin = cfg.sample_count = 0
    px = torch.empty((size[1], size[0], 3), device="cuda")
    L.sums_finalize_device(whole.data_ptr(), *size, 1.0, px.data_ptr())
    torch.cuda.synchronize()
    np.testing.assert_array_equal(px.cpu().numpy(), sc.render(cfg)[0])
    sc.close()


@pytest.mark.parametrize("build", ["spheres", "box_room", "zoo"])
@pytest.mark.parametrize("size", [(1, 1), (9, 5), (37, 21)])
def test_aov_builds_at_ragged_sizes_match_the_oracle(build, size):
    """Each build of the AOV kernel over partial 8x4 tiles, by the rules of the other AOV tests."""
    import oracle as O
    world, cfg = (W.random_spheres if build == "spheres" else SCENES[build][0])(*(size if build == "spheres" else ()))
    cfg.width, cfg.height = size
    sc = L.GpuScene(world)
    got = sc.render_aov(cfg)
    sc.close()
    want = O.OracleScene(world).render_aov(cfg, mode=O.MODE_KEYED)
    if size == (1, 1):
        return                                   # a 1x1 frame's ray has no finite direction
    hit = (got[0] > 0) & (want[0] > 0)
    assert ((got[0] > 0) == (want[0] > 0)).mean() >= 0.995
    assert (np.abs(got[0] - want[0])[hit] <= 5e-4 * want[0][hit]).mean() >= 0.98
    assert (np.abs(got[1].astype(int) - want[1].astype(int)) <= 1).mean() >= 0.98
    assert (np.abs(got[2].astype(int) - want[2].astype(int)) <= 1).mean() >= 0.96


@pytest.mark.parametrize("n", [507, 508, 1000])
def test_quad_builds_equal_the_other_modes(n):
    """Quad scenes of both sides of 512 quads (four are the lights), from which warps turn to the leaves
    early: the wavefront and the batched megakernel, which never do, give the same image."""
    from luminara_b200 import abi
    world, cfg = W.diff_quads(61, 35, 4, n_quads=n)
    sc = L.GpuScene(world)
    assert sc.info()["prims"] == n + 4
    img, _ = sc.render(cfg)
    for mode in (abi.BATCH_WAVEFRONT, abi.BATCH_MEGAKERNEL, abi.BATCH_STREAMS):
        batch = L.Batch([sc], [cfg], config={"mode": mode})
        np.testing.assert_array_equal(batch.render()[0][0], img)
        batch.close()
    sc.close()


@pytest.mark.parametrize("build", ["spheres", "box_room", "zoo"])
def test_aov_crops_equal_the_frame(build):
    """AOVs of crops with one live lane, a row, a column and partial tiles, against the whole frame's.  A
    1x1 frame's ray has no finite direction (its pixel grid has no width), so it meets nothing."""
    world, cfg = (W.random_spheres if build == "spheres" else SCENES[build][0])(*((64, 48) if build == "spheres" else ()))
    sc = L.GpuScene(world)
    frame = sc.render_aov(cfg)
    assert all(p.any() for p in frame)
    for crop in ((0, 0, 1, 1), (33, 20, 1, 1), (40, 30, 1, 9), (5, 47, 17, 1), (7, 3, 9, 5), (40, 30, 24, 18)):
        cfg.crop = crop
        x, y, w, h = crop
        for part, whole in zip(sc.render_aov(cfg), frame):
            np.testing.assert_array_equal(part, whole[y:y + h, x:x + w])
    cfg.crop = None
    cfg.width = cfg.height = 1
    assert not any(p.any() for p in sc.render_aov(cfg))
    sc.close()


def _sampled_scene(build):
    if build == "quads":
        return W.diff_quads(64, 48, 20, n_quads=40)
    if build == "spheres":
        return W.random_spheres(64, 48, 20)
    if build == "mixed":
        return W.uneven_scene(np.random.default_rng(1), 300, 64, 48, 20)
    return SCENES[build][0]()


SAMPLED = ["spheres", "box_room", "quads", "mesh", "zoo", "mixed"]


@pytest.mark.parametrize("threshold", [0.0, 0.05])
@pytest.mark.parametrize("build", SAMPLED)
def test_adaptive_crops_equal_the_frame(build, threshold):
    """Every build of the adaptive kernel, bit for bit: a pixel's samples and its stop do not depend on the
    pixels that share its pool, so crops with 1 to 32 pixels per tile equal the whole frame.  25 strata
    in rounds of 16 and 9."""
    world, cfg = _sampled_scene(build)
    cfg.samples_per_pixel, cfg.adaptive, cfg.adaptive_threshold = 20, True, threshold
    sc = L.GpuScene(world)
    frame, st = sc.render(cfg)
    assert (st.paths == 25 * 64 * 48) == (threshold == 0.0) and st.paths >= 16 * 64 * 48
    for x, y, w, h in ((0, 0, 1, 1), (33, 20, 1, 1), (7, 3, 9, 5), (50, 41, 7, 4), (11, 30, 3, 18), (0, 5, 64, 3)):
        cfg.crop = (x, y, w, h)
        np.testing.assert_array_equal(sc.render(cfg)[0], frame[y:y + h, x:x + w])
    sc.close()


@pytest.mark.parametrize("build", SAMPLED)
def test_time_limit_that_does_not_run_out_equals_the_render(build):
    """Every time-limited build, its pool one tile's strata, gives the plain render's sums."""
    world, cfg = _sampled_scene(build)
    cfg.width, cfg.height, cfg.samples_per_pixel = 37, 21, 20
    sc = L.GpuScene(world)
    plain, _ = sc.render(cfg)
    cfg.time_limit = 1000.0
    np.testing.assert_array_equal(sc.render(cfg)[0], plain)
    sc.close()
