"""Staged, gated and plain sweeps of a launch shape give the same bits at every color size, although each
picks between its register-capped and its uncapped build by occupancy.  At 16 lanes the uncapped builds
evaluate a lane's first triangle and first hinge side by side, and add them in the capped builds' order."""

import pytest
import torch

from newton_b200 import scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


# 16 lanes of 128 threads: colors of 6,400 / 7,396 / 7,921 / 8,464 vertices, below, between and above one wave of
# the builds (72 to 80 registers)
@pytest.mark.parametrize("n, lanes, block, kd", [(160, 16, 128, 1e-3), (172, 16, 128, 1e-3), (178, 16, 128, 1e-3),
                                                 (184, 16, 128, 1e-3), (178, 16, 256, 1e-3), (178, 2, 128, 1e-3),
                                                 (178, 16, 128, 0.0)])
def test_staged_gated_and_plain_sweeps_give_the_same_bits(n, lanes, block, kd):
    material = dict(tri_ke=1.0e4, tri_ka=1.0e4, tri_kd=kd, edge_ke=1.0e-2, edge_kd=kd)
    model, q0 = scenes.single_cloth(n=n, side=2.0, seed=1, ground=None, height=0.0, vertical=True, material=material)
    results = []
    for staged, gated in ((False, False), (True, False), (False, True), (True, True)):
        solver = SolverVBD(model, iterations=4)
        solver.set_launch(lanes, block)
        if staged:
            solver.set_staged_sweep(True)
            assert solver.staged_sweep_info()["active"]
        if gated:  # never reached: every step runs to the cap
            solver.set_residual_gate(1e-20, max_iterations=4, residual="sweep")
        a, b = model.state(), model.state()
        a.particle_q.copy_(torch.from_numpy(q0).cuda())
        for _ in range(3):
            solver.step(a, b, None, None, DT)
            a, b = b, a
        if gated:
            assert solver.gate_stats()["last_iterations"] == 4
        results.append(a.particle_q.clone())
    for other in results[1:]:
        assert torch.equal(results[0], other)


@pytest.mark.parametrize("n, lanes", [(128, 16), (130, 8), (182, 8), (184, 4)])  # colors of 4,096 / 4,225 / 8,281 / 8,464
def test_default_lanes_at_the_lines(n, lanes):
    model, _ = scenes.draped_cloth(n=n, seed=0)
    largest = max(len(g) for g in model.particle_color_groups)
    assert (largest <= 4144) == (lanes == 16) and (largest <= 8288) == (lanes >= 8)
    assert SolverVBD(model).launch_info()["lanes_per_vertex"] == lanes
