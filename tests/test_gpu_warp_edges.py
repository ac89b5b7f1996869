"""GPU test of calls whose rays or pixels do not fill whole warps.

The traversal walks a warp's rays together, lanes without a ray following along, so the results
of a small or ragged call must equal those of the same rays and pixels inside a larger one, bit
for bit: ray sets around the warp (32) and block (128) sizes, and crops smaller than an 8x4 tile.
"""
import numpy as np
import pytest

import luminara_b200 as L
from luminara_b200 import workloads as W

from .helpers import random_rays, to_gpu_rays

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
