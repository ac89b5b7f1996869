"""GPU test of the adjoint's staging buffer, which one call leaves for the next: calls of different
sizes, on scenes of their own and on two threads at once, give the gradients of a call by itself."""
import os
import subprocess
import sys
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


def test_staging_goes_back_with_the_last_scene():
    """Free device memory after a backward call: less by the kept buffer while a scene lives, and what it
    was before (the scenes' pool keeps a few MB) once the last one is closed."""
    code = """
import numpy as np, torch
import luminara_b200 as L
from luminara_b200 import workloads as W
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
def backward(world, cfg):
    sc = L.GpuScene(world)
    sc.backward(cfg, np.full(cfg.out_shape(), 1e-3, np.float32), world.light_material_indices())
    return sc
backward(*W.diff_quads(16, 8, 4)).close()          # the context, the kernels and the pool
before = free()
world, cfg = W.diff_quads(256, 256, 16)
a, b = L.GpuScene(world), backward(world, cfg)
staged = before - free()
b.close()
kept = before - free()
a.close()
print(staged, kept, before - free())
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    staged, kept, left = map(int, r.stdout.split())
    # 256 * 256 * 16 paths of at least 48 + 64 bytes
    assert staged > 100 << 20 and kept > 100 << 20
    assert left <= 64 << 20
