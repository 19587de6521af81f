"""Self-contact on a GPU without room for the full pair tables: the solver is created with smaller ones,
the rows that do not fit are evaluated from the detection lists, and forces and truncation stay the same."""

import gc

import numpy as np
import pytest
import torch

from newton_b200 import scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


def _evaluate(model, q, qd):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=0.003,
                       particle_self_contact_margin=0.0045)
    used = before - torch.cuda.mem_get_info()[0]
    state = model.state()
    state.particle_q.copy_(torch.from_numpy(q).cuda())
    state.particle_qd.copy_(torch.from_numpy(qd).cuda())
    solver.forward(state, None, DT)
    x = solver.positions().cpu().numpy()
    r = solver.residual(None, DT, per_vertex=True)[1].cpu().numpy()
    assert solver.status()["self_contact_overflow"] == 0
    return used, x, r


def test_smaller_tables_where_the_full_ones_do_not_fit():
    n = 400
    model, q0 = scenes.single_cloth(n=n, side=2.0, seed=0, pin_top_corners=False, ground=None, z_noise=0.0)
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1.0e3, 1.0e-2, 0.2
    q = q0.copy()
    right = q[:, 0] > 0.0
    q[right, 0] = -q[right, 0]
    q[right, 2] += 0.0025
    qd = np.random.default_rng(1).uniform(-0.6, 0.6, q.shape).astype(np.float32)  # 1 mm in a step
    used, x, r = _evaluate(model, q, qd)
    tables = n * n * (96 * 16 + 24 * 48)
    assert used > tables
    for short in (0.5, 0.95):  # of the tables' bytes: what the GPU lacks
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        room = int(used - short * tables) + (32 << 20)
        filler = torch.empty(max(torch.cuda.mem_get_info()[0] - room, 0), dtype=torch.uint8, device="cuda")
        small, xs, rs = _evaluate(model, q, qd)
        del filler
        assert small < used - 0.4 * tables
        # the same pairs, planes and forces; planes from the lists and from the table's heights round
        # differently (1e-6 of the 1 mm moves and positions of 1 m: 2e-7), the sums run in another order
        assert np.abs(x - xs).max() <= 5e-7
        assert np.abs(r - rs).max() <= 1e-4 * r.max()
    torch.cuda.empty_cache()
