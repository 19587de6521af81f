"""The pair tables of cloth self-contact (entries per vertex, flat division planes) against the CPU
oracle, with the pairs inside the tables' capacity and far beyond it: rows that do not fit are
evaluated from the detection lists, and both must agree with the oracle.  Rows beyond the rank sort's
width (64 entries) are sorted by one lane."""

import numpy as np
import pytest
import torch

import oracle
from newton_b200 import scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu

DT = 1.0 / 600.0
RADIUS, BUFFERS = 0.004, (64, 256)


def _folded(n=24, side=0.5, gap=0.003):
    model, q0 = scenes.single_cloth(n=n, side=side, seed=0, pin_top_corners=False, ground=None, z_noise=0.0)
    q = q0.astype(np.float64).copy()
    right = q[:, 0] > 0.0
    q[right, 0] = -q[right, 0]
    q[right, 2] += gap
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1.0e3, 1.0e-2, 0.2
    return model, q.astype(np.float32)


def _around(x, n=24, rings=2):
    """The largest value within two rows and columns of each vertex of the n x n cloth."""
    padded = np.pad(x.reshape(n, n), rings)
    shifts = [padded[r:r + n, c:c + n] for r in range(2 * rings + 1) for c in range(2 * rings + 1)]
    return np.max(shifts, axis=0).reshape(-1)


def test_rows_beyond_the_rank_sort_are_ordered():
    model, q = _folded()
    solver = SolverVBD(model, iterations=1, particle_enable_self_contact=True, particle_self_contact_radius=RADIUS,
                       particle_self_contact_margin=0.05, particle_vertex_contact_buffer_size=256,
                       particle_edge_contact_buffer_size=512)
    orc = oracle.VBDOracle(model, "f32")
    orc.set_self_contact(radius=RADIUS, margin=0.05, vertex_buffer=256, edge_buffer=512, rest_q=model.particle_q)
    vc, vl, ec, el = solver.self_contact_detect(torch.from_numpy(q).cuda())
    ovc, ovl, oec, oel, dropped = orc.self_contact_detect(q)
    assert dropped == 0 and int(ec.max()) > 64
    np.testing.assert_array_equal(vc, ovc)
    np.testing.assert_array_equal(vl, ovl)
    np.testing.assert_array_equal(ec, oec)
    np.testing.assert_array_equal(el, oel)


@pytest.mark.parametrize("margin, beyond", [(0.006, False), (0.030, True)])
def test_tables_within_and_beyond_their_capacity(margin, beyond):
    model, q = _folded()
    kw = dict(particle_enable_self_contact=True, particle_self_contact_radius=RADIUS,
              particle_self_contact_margin=margin, particle_vertex_contact_buffer_size=BUFFERS[0],
              particle_edge_contact_buffer_size=BUFFERS[1])
    solver = SolverVBD(model, iterations=5, **kw)
    orc = oracle.VBDOracle(model, "f32")
    orc.set_self_contact(radius=RADIUS, margin=margin, vertex_buffer=BUFFERS[0], edge_buffer=BUFFERS[1],
                         rest_q=model.particle_q)
    vc, vl, ec, el = solver.self_contact_detect(torch.from_numpy(q).cuda())
    ovc, ovl, oec, oel, dropped = orc.self_contact_detect(q)
    assert dropped == 0
    np.testing.assert_array_equal(vc, ovc)
    np.testing.assert_array_equal(vl, ovl)
    np.testing.assert_array_equal(ec, oec)
    np.testing.assert_array_equal(el, oel)
    # the capacities are 96 entries and 24 pairs per vertex on average; a pair has four entries
    V = model.particle_count
    pairs = int(vc.sum()) + int(ec.sum()) // 2
    assert (pairs > 24 * V) == beyond and (4 * pairs > 96 * V) == beyond
    exact = oracle.VBDOracle(model, "f64")
    exact.set_self_contact(radius=RADIUS, margin=margin, vertex_buffer=BUFFERS[0], edge_buffer=BUFFERS[1],
                           rest_q=model.particle_q)
    a, b = model.state(), model.state()
    a.particle_q.copy_(torch.from_numpy(q).cuda())
    for _ in range(3):
        q_in, qd_in = a.particle_q.cpu().numpy().copy(), a.particle_qd.cpu().numpy().copy()
        solver.step(a, b, None, None, DT)
        _, q_ref, _ = orc.step(q_in, qd_in, None, DT, 5)
        _, q_64, _ = exact.step(q_in, qd_in, None, DT, 5)
        # the parity tolerance of a step, and at vertices where pushing out of the 3 mm overlap is
        # ill-conditioned (a wider margin lets them move farther in one step), what FP32 itself is off by:
        # four times the FP32 oracle's distance from the FP64 one at the vertex or two rings around it,
        # but never more than 1% of the radius (a missing contact moves a vertex by 1 mm and more)
        bound = np.minimum(1e-5 + 4.0 * _around(np.abs(q_ref - q_64).max(axis=1)), 0.01 * RADIUS)
        assert (np.abs(b.particle_q.cpu().numpy() - q_ref).max(axis=1) <= bound).all()
        a, b = b, a
    st = solver.status()
    assert st["self_contact_overflow"] == 0 and st["nonfinite_updates"] == 0
