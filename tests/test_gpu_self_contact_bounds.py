"""The early rejection of the self-contact force pass (a pair's distance at the detected positions less
what its vertices have moved since) never changes a result: the forces equal, bit for bit, those of the
same detection without displacement bounds (``self_contact_detect`` gives the pass none)."""

import numpy as np
import pytest
import torch

from newton_b200 import ModelBuilder, scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


def _layers(n, cell, gap, shift=0.0):
    """Two square cloths of n x n vertices, the upper one turned by 90 degrees, shifted and lifted by gap."""
    b = ModelBuilder()
    verts, tris = ModelBuilder.grid_mesh(n - 1, n - 1, cell, cell)
    for k in range(2):
        b.add_cloth_mesh(pos=(0.0, 0.0, 0.0), rot=(0.0, 0.0, 0.0, 1.0), scale=1.0, vel=(0.0, 0.0, 0.0), vertices=verts,
                         indices=tris, density=0.1, tri_ke=1.0e3, tri_ka=1.0e3, tri_kd=0.0, edge_ke=0.0, edge_kd=0.0)
    b.color()
    model = b.finalize()
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1.0e3, 1.0e-2, 0.2
    q = model.particle_q.astype(np.float64).copy()
    side = cell * (n - 1)
    up = np.arange(q.shape[0]) >= n * n
    x, y = q[up, 0].copy(), q[up, 1].copy()
    q[up, 0], q[up, 1] = side - y + shift, x + shift
    q[up, 2] += gap
    return model, q.astype(np.float32), up


def _residuals(model, q, qd, radius, margin):
    """(after forward, after detecting again at the step's start, after detecting at the iterate)"""
    solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=radius,
                       particle_self_contact_margin=margin, particle_vertex_contact_buffer_size=128,
                       particle_edge_contact_buffer_size=256)
    state = model.state()
    state.particle_q.copy_(torch.from_numpy(q).cuda())
    state.particle_qd.copy_(torch.from_numpy(qd).cuda())
    solver.forward(state, None, DT)
    moved = solver.positions()
    out = [solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()]
    for at in (state.particle_q, moved):
        solver.self_contact_detect(at)
        out.append(solver.residual(None, DT, per_vertex=True)[1].cpu().numpy())
    assert solver.status()["self_contact_overflow"] == 0
    return out


def test_detection_at_other_positions_than_the_iterate():
    """The layers are 3 mm apart at the step's start (radius 2 mm) and 1.5 mm apart at the iterate: the
    forces are the same whether the pairs were detected at the former or at the latter."""
    model, q, up = _layers(12, 0.02, 0.003, 0.006)
    qd = np.zeros_like(q)
    qd[up, 2] = -0.0015 / DT
    first, again, there = _residuals(model, q, qd, 0.002, 0.004)
    solo, _, _ = _residuals(model, q + np.where(up, 0.1, 0.0)[:, None].astype(np.float32), qd, 0.002, 0.004)
    assert np.abs(first - solo).max() > 1e3 * np.abs(solo).max()  # (contact forces are there)
    np.testing.assert_array_equal(first, again)
    # other lists, other order of the same FP32 sums
    np.testing.assert_allclose(again, there, rtol=1e-4, atol=1e-5 * there.max())


def test_warm_start_from_another_base_than_the_detected_one():
    """``warm_start`` puts the iterate at the step's start (3 mm apart, radius 3.2 mm) plus its displacement,
    after a detection at the iterate (4 mm apart) that made those positions the base."""
    model, q, up = _layers(12, 0.02, 0.003, 0.006)
    qd = np.zeros_like(q)
    qd[up, 2] = 0.001 / DT

    def residuals(q):
        solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=0.0032,
                           particle_self_contact_margin=0.005)
        state = model.state()
        state.particle_q.copy_(torch.from_numpy(q).cuda())
        state.particle_qd.copy_(torch.from_numpy(qd).cuda())
        solver.forward(state, None, DT)
        base = solver.positions()
        solver.begin_iteration()
        solver.warm_start(torch.zeros_like(state.particle_q))
        assert torch.equal(solver.positions(), state.particle_q)
        first = solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()
        solver.self_contact_detect(base)
        return first, solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()

    first, again = residuals(q)
    solo, _ = residuals(q + np.where(up, 0.1, 0.0)[:, None].astype(np.float32))
    assert np.abs(first - solo).max() > 2.0 * np.abs(solo).max()  # (contact forces are there)
    np.testing.assert_array_equal(first, again)


@pytest.mark.parametrize("stretch", [0.04, 0.0, -0.04])
@pytest.mark.parametrize("cell", [0.0031, 0.0032])
def test_edges_that_cross_the_length_threshold(cell, stretch):
    """Edges below sqrt(edge_parallel_epsilon) = 3.16 mm count as points, so stretching one beyond it
    brings a crossing pair from its first endpoints' distance (2.4 mm) to the crossing's (1 mm)."""
    model, q, up = _layers(7, cell, 0.001, 0.5 * cell)
    centre = q.mean(axis=0)
    qd = (stretch / DT * (q - centre)).astype(np.float32)
    qd[:, 2] = 0.0
    first, again, _ = _residuals(model, q, qd, 0.002, 0.003)
    np.testing.assert_array_equal(first, again)


def test_thin_triangles_and_near_parallel_edges():
    """Random thin cloths (aspect down to 1e-4) across one another, moved at random: where FP32 misses a
    pair's closest points, its bound must not reject what the direct test takes."""
    rng = np.random.default_rng(7)
    model, q, up = _layers(5, 0.004, 0.0025, 0.0)
    for k in range(12):
        squeeze = 10.0 ** rng.uniform(-4.0, 0.0)
        p = q.astype(np.float64).copy()
        p[:, 1] *= squeeze
        p[up, 1] += rng.uniform(-1.0, 1.0) * 0.002
        p = p.astype(np.float32)
        qd = (rng.uniform(-1.0, 1.0, size=p.shape) * 0.0012 / DT).astype(np.float32)
        solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=0.002,
                           particle_self_contact_margin=0.003, particle_vertex_contact_buffer_size=128,
                           particle_edge_contact_buffer_size=256)
        state = model.state()
        state.particle_q.copy_(torch.from_numpy(p).cuda())
        state.particle_qd.copy_(torch.from_numpy(qd).cuda())
        solver.forward(state, None, DT)
        first = solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()
        solver.self_contact_detect(state.particle_q)
        again = solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()
        np.testing.assert_array_equal(first, again)
        assert solver.status()["self_contact_overflow"] == 0


def test_warm_start_beyond_the_bound_is_clamped_by_the_first_color():
    """``warm_start`` may move vertices beyond margin * relaxation / 2; the truncation after the first
    color brings every vertex back to it, whatever its color."""
    model, q0 = scenes.single_cloth(n=16, side=1.0, seed=0, pin_top_corners=False, ground=None)
    margin, bound = 0.004, 0.004 * 0.85 * 0.5
    solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=0.002,
                       particle_self_contact_margin=margin, particle_collision_detection_interval=-1)
    state = model.state()
    state.particle_q.copy_(torch.from_numpy(q0).cuda())
    solver.forward(state, None, DT)
    delta = np.zeros_like(q0)
    delta[:, 2] = 0.01
    solver.warm_start(torch.from_numpy(delta).cuda())
    assert np.linalg.norm(solver.positions().cpu().numpy() - q0, axis=1).min() > bound
    solver.begin_iteration()
    solver.sweep_color(0, None, DT)
    x = solver.positions().cpu().numpy()
    assert np.linalg.norm(x - q0, axis=1).max() <= bound * (1.0 + 1e-4)
