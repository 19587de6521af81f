"""Sixteen lanes per vertex, where a lane takes its first triangle and its first hinge together: fans
whose hub owns fewer, as many and more triangles than there are lanes, against the CPU oracle."""

import numpy as np
import pytest
import torch

import oracle
from newton_b200.builder import ModelBuilder
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


@pytest.mark.parametrize("damping", [0.0, 1.0e-3])
@pytest.mark.parametrize("triangles", [1, 2, 8, 15, 16, 17, 33])
def test_fans_match_the_oracle(triangles, damping):
    angle = np.arange(triangles + 1) * (1.6 * np.pi / triangles if triangles > 2 else 0.9)
    rim = np.stack([0.1 * np.cos(angle), 0.1 * np.sin(angle), 0.01 * np.cos(3.0 * angle)], axis=1)
    k = np.arange(1, triangles + 1)
    builder = ModelBuilder()
    builder.add_cloth_mesh(pos=(0.0, 0.0, 1.0), rot=(0.0, 0.0, 0.0, 1.0), scale=1.0, vel=(0.0, 0.0, 0.0),
                           vertices=np.concatenate([np.zeros((1, 3)), rim]),
                           indices=np.stack([np.zeros_like(k), k, k + 1], axis=1).reshape(-1), density=0.2,
                           tri_ke=1.0e3, tri_ka=1.0e3, tri_kd=damping, edge_ke=5.0e-2, edge_kd=damping)
    builder.color(include_bending=True)
    model = builder.finalize("cuda:0")
    rng = np.random.default_rng(triangles)
    q = (np.asarray(model.particle_q, dtype=np.float32).reshape(-1, 3)
         + rng.uniform(-2e-3, 2e-3, (triangles + 2, 3))).astype(np.float32)
    qd = rng.uniform(-0.2, 0.2, q.shape).astype(np.float32)
    solver = SolverVBD(model, iterations=6, lanes_per_vertex=16, block_size=128)
    a, b = model.state(), model.state()
    a.particle_q.copy_(torch.from_numpy(q).cuda())
    a.particle_qd.copy_(torch.from_numpy(qd).cuda())
    solver.step(a, b, None, None, DT)
    _, ref, _ = oracle.VBDOracle(model, "f32").step(q, qd, None, DT, 6)
    # the parity tolerance of a step
    assert np.abs(b.particle_q.cpu().numpy() - ref).max() <= 1e-5
