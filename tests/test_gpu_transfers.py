"""GPU test of the shared staging buffers: ray sets and frames of sizes around the rule's limits
(csrc/staging_rule.h), by one thread and by three at once, give the bytes of a set sent in small pieces,
which never takes the buffers."""
import threading

import numpy as np
import pytest

import luminara_b200 as L
from luminara_b200 import workloads as W

pytestmark = pytest.mark.gpu

# 48 bytes up and down per ray: around 3 MB, above 8 MB, above four 8 MB chunks with a remainder
SIZES = (1, 65_535, 65_537, 180_000, 760_001)


def _rays(world, n, seed):
    rng = np.random.default_rng(seed)
    return L.make_rays(np.tile(world.camera.look_from, (n, 1)), rng.normal(size=(n, 3)) + np.array([0.0, -0.3, -2.0]))


def test_transfers_of_all_sizes_and_threads():
    world, cfg = W.random_spheres(width=1280, height=720, spp=1)
    sets = [_rays(world, n, k) for k, n in enumerate(SIZES)]
    sc = L.GpuScene(world)
    cut = 20_000                                   # under 1 MB
    want = [np.concatenate([sc.intersect(r[k:k + cut]) for k in range(0, len(r), cut)]) for r in sets]
    occ = [np.concatenate([sc.occluded(r[k:k + cut]) for k in range(0, len(r), cut)]) for r in sets]
    frame, _ = sc.render(cfg)
    errors = []

    def work(turn):
        mine = L.GpuScene(world)
        try:
            for step in range(2 * len(sets)):
                k = (step + turn) % len(sets)
                if mine.intersect(sets[k]).tobytes() != want[k].tobytes():
                    errors.append(("intersect", SIZES[k], turn))
                if not np.array_equal(mine.occluded(sets[k]), occ[k]):
                    errors.append(("occluded", SIZES[k], turn))
                if turn and not np.array_equal(mine.render(cfg)[0], frame):
                    errors.append(("render", turn))
        finally:
            mine.close()

    work(0)
    threads = [threading.Thread(target=work, args=(t,)) for t in (1, 2, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    sc.close()
    assert errors == []
