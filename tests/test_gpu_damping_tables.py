"""Sweeps with the step-start metrics and angles from the once-per-step tables: membrane and bending
damping, and triangles stretched beyond the clamp of the area term (the branch that unstretched
cloth skips), against the CPU oracle; the allocation-free step, which evaluates the step-start
positions in the sweep instead, gives the same bits."""

import ctypes

import numpy as np
import pytest
import torch

import oracle
from newton_b200 import _lib, scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


def _scene(tri_kd, edge_kd, stretch):
    material = dict(tri_ke=5.0e3, tri_ka=5.0e3, tri_kd=tri_kd, edge_ke=5.0e-2, edge_kd=edge_kd)
    model, q0 = scenes.single_cloth(n=37, side=0.8, seed=3, pin_top_corners=True, ground=None, height=0.9,
                                    vertical=True, material=material, z_noise=2e-3)
    q = q0.copy()
    q[:, 0] *= stretch
    q[:, 2] = 0.9 + (q[:, 2] - 0.9) * stretch
    rng = np.random.default_rng(4)
    qd = rng.uniform(-0.3, 0.3, q.shape).astype(np.float32) * (model.particle_mass > 0)[:, None]
    return model, q.astype(np.float32), qd


def _states(model, q, qd):
    a, b = model.state(), model.state()
    a.particle_q.copy_(torch.from_numpy(q).cuda())
    a.particle_qd.copy_(torch.from_numpy(qd).cuda())
    return a, b


@pytest.mark.parametrize("lanes", [0, 1, 2, 4, 8, 16])
@pytest.mark.parametrize("tri_kd, edge_kd, stretch", [(0.0, 0.0, 1.3), (1e-2, 0.0, 1.3), (1e-2, 1e-3, 1.0), (0.0, 1e-3, 1.0)])
def test_damped_and_stretched_steps_match_the_oracle(tri_kd, edge_kd, stretch, lanes):
    model, q, qd = _scene(tri_kd, edge_kd, stretch)
    solver = SolverVBD(model, iterations=6, lanes_per_vertex=lanes if lanes else -1, block_size=128)
    a, b = _states(model, q, qd)
    solver.step(a, b, None, None, DT)
    _, ref, _ = oracle.VBDOracle(model, "f32").step(q, qd, None, DT, 6)
    # the parity tolerance of a step
    assert np.abs(b.particle_q.cpu().numpy() - ref).max() <= 1e-5
    if lanes > 0:
        staged = SolverVBD(model, iterations=6, lanes_per_vertex=lanes, block_size=128)
        staged.set_staged_sweep(True)
        c, d = _states(model, q, qd)
        staged.step(c, d, None, None, DT)
        assert torch.equal(b.particle_q, d.particle_q)


@pytest.mark.parametrize("tri_kd, edge_kd", [(1e-2, 0.0), (1e-2, 1e-3)])
def test_step_without_tables_gives_the_same_bits(tri_kd, edge_kd):
    model, q, qd = _scene(tri_kd, edge_kd, 1.0)
    solver = SolverVBD(model, iterations=6, lanes_per_vertex=4, block_size=128)
    a, b = _states(model, q, qd)
    solver.step(a, b, None, None, DT)
    c, d = _states(model, q, qd)
    lib = _lib.load()
    _lib.check(lib.vbd_step_static(model.device_model().handle, _lib.ptr(c.particle_q), _lib.ptr(c.particle_qd),
                                   _lib.ptr(c.particle_f), _lib.ptr(d.particle_q), _lib.ptr(d.particle_qd), None,
                                   ctypes.c_float(DT), 6, ctypes.c_float(1e-2), solver._stream()))
    assert torch.equal(b.particle_q, d.particle_q) and torch.equal(b.particle_qd, d.particle_qd)
