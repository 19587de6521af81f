"""The room of the record staging (4 lanes) at the most shared memory a launch gets by default: 48 KB,
which the kernel's own static part comes out of."""

import numpy as np
import pytest
import torch

from newton_b200 import ModelBuilder
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


def _fans(bending):
    """64 separate fans, their hubs one color (one block of 256 threads at 4 lanes): 56 of 16 triangles and
    8 of 15, the last one with bending: 1,016 triangle and 15 hinge records, 49,152 bytes."""
    b = ModelBuilder()
    groups = [[], [], [], []]
    for k in range(64):
        n = 16 if k < 56 else 15
        start = b.particle_count
        t = 2.0 * np.pi * np.arange(n) / n
        verts = np.concatenate([np.zeros((1, 3)), 0.05 * np.stack([np.cos(t), np.sin(t), 0.1 * np.cos(3 * t)], axis=1)])
        tris = np.array([[0, 1 + i, 1 + (i + 1) % n] for i in range(n)])
        b.add_cloth_mesh(pos=(0.2 * (k % 8), 0.2 * (k // 8), 0.0), rot=(0.0, 0.0, 0.0, 1.0), scale=1.0,
                         vel=(0.0, 0.0, 0.0), vertices=verts, indices=tris.reshape(-1), density=0.1, tri_ke=1.0e3,
                         tri_ka=1.0e3, tri_kd=1.0e-3, edge_ke=1.0e-2 if bending and k == 63 else 0.0, edge_kd=0.0)
        groups[0].append(start)
        for i in range(n):
            groups[1 + (i % 2 if n == 16 else i % 3)].append(start + 1 + i)
    b.set_coloring([np.array(g, dtype=np.int32) for g in groups])
    return b.finalize()


@pytest.mark.parametrize("bending", [True, False])
def test_a_block_whose_records_fill_the_default_shared_memory(bending):
    model = _fans(bending)
    results = []
    for block in (256, 128):
        solver = SolverVBD(model, iterations=5)
        solver.set_launch(4, block)
        a, b = model.state(), model.state()
        rng = np.random.default_rng(0)
        a.particle_q.add_(torch.from_numpy(rng.uniform(-1e-3, 1e-3, a.particle_q.shape).astype(np.float32)).cuda())
        for _ in range(3):
            solver.step(a, b, None, None, DT)
            a, b = b, a
        st = solver.status()
        assert st["timeouts"] == 0 and st["nonfinite_updates"] == 0
        results.append(a.particle_q.clone())
    assert torch.isfinite(results[0]).all() and torch.equal(results[0], results[1])
