"""The force residual and the staged sweeps after a resident step of a damped model: both damp against
the positions at that step's start, as they do after a step of one launch per color."""

import pytest
import torch

from newton_b200 import scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0
MATERIALS = {
    "membrane": dict(tri_ke=1.0e4, tri_ka=1.0e4, tri_kd=1.0e-3, edge_ke=1.0e-2, edge_kd=0.0),
    "membrane_and_bending": dict(tri_ke=1.0e4, tri_ka=1.0e4, tri_kd=1.0e-3, edge_ke=1.0e-2, edge_kd=1.0e-3),
}


@pytest.mark.parametrize("material", list(MATERIALS))
def test_residual_and_sweeps_after_resident_steps(material):
    model, q0 = scenes.single_cloth(n=40, side=1.0, seed=4, ground=None, height=0.0, vertical=True,
                                    material=MATERIALS[material])
    out = []
    for resident in (True, False):
        solver = SolverVBD(model, iterations=10, lanes_per_vertex=4, block_size=128, resident_step=resident)
        a, b = model.state(), model.state()
        a.particle_q.copy_(torch.from_numpy(q0).cuda())
        for _ in range(4):
            solver.step(a, b, None, None, DT)
            a, b = b, a
        assert solver.step_kernel_info()["resident"] == resident
        q = solver.positions().clone()
        _, r = solver.residual(None, DT, per_vertex=True)
        r = r.clone()
        solver.iterate(None, DT, 1)
        out.append((q, r, solver.positions().clone()))
        assert solver.status()["timeouts"] == 0
    (qa, ra, xa), (qb, rb, xb) = out
    # the two step kernels round alike up to single ulps of positions below 2 m (1.2e-7 m); a vertex's
    # force moves by its stiffness, about 4 (tri_ke + tri_ka) = 8e4 N/m, against m|g| of 0.1 kg/m^2 on
    # a cell of (1/39 m)^2 = 6.4e-4 N: a residual difference of 8e4 / 6.4e-4 per metre
    dq = float((qa - qb).abs().max())
    dr, dx = float((ra - rb).abs().max()), float((xa - xb).abs().max())
    print(f"{material}: |dq| {dq:.3e} |dr| {dr:.3e} of {float(rb.max()):.3e} |dx| {dx:.3e}")
    assert dq <= 1e-6 and dx <= 1e-6
    assert dr <= 1e-5 * float(rb.max()) + dq * 8.0e4 / 6.4e-4
