"""GPU test of the adjoint's staging buffer, which one call leaves for the next: calls of different
sizes, on scenes of their own and on two threads at once, give the gradients of a call by itself."""
import threading

import numpy as np
import pytest

import luminara_b200 as L
from luminara_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _backward(size):
    world, cfg = W.diff_quads(*size)
    sc = L.GpuScene(world)
    dl = np.full(cfg.out_shape(), 1e-3, np.float32)
    grads = sc.backward(cfg, dl, world.light_material_indices())[:3]
    sc.close()
    return [g.astype(np.float64) for g in grads]


@pytest.mark.parametrize("sizes", [((16, 8, 4), (96, 64, 16)), ((96, 64, 16), (96, 64, 16)),
                                   ((133, 77, 16), (8, 4, 1))])
def test_staging_is_shared_by_sizes_and_threads(sizes):
    want = [_backward(s) for s in sizes]
    got = [[] for _ in sizes]

    def work(k):
        for _ in range(6):
            got[k].append(_backward(sizes[k]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(sizes)):
        assert len(got[k]) == 6
        for grads in got[k]:
            for g, w in zip(grads, want[k]):
                # float sums of up to 133 * 77 * 16 * 6 = 1e6 terms in another order: sqrt(n) * 6e-8
                # of the terms' size, with a factor 16 for cancellation among them
                assert np.linalg.norm(g - w) <= 1e-3 * np.linalg.norm(w) + 1e-12
