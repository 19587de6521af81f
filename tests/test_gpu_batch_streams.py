"""``SolverVBD.step_batch`` runs small independent solvers beside one another: the same bits as one
``step`` per solver in order, ordered with the caller's stream before and after, and in order when
one entry reads what another writes or a solver appears twice."""

import pytest
import torch

from newton_b200 import CollisionPipeline, scenes
from newton_b200.solvers import SolverVBD

pytestmark = pytest.mark.gpu
DT = 1.0 / 600.0


def _entries(sizes):
    out = []
    for k, n in enumerate(sizes):
        model, q0 = scenes.draped_cloth(n=n, seed=k, height=0.902)
        pipe = CollisionPipeline(model, soft_contact_margin=5e-3)
        a, b = model.state(), model.state()
        a.particle_q.copy_(torch.from_numpy(q0).cuda())
        out.append([SolverVBD(model, iterations=4), pipe, pipe.contacts(), a, b])
    return out


def _run(entries, steps, batch, stream):
    with torch.cuda.stream(stream):
        for _ in range(steps):
            for e in entries:
                e[1].collide(e[3], e[2])
            if batch:
                SolverVBD.step_batch([e[0] for e in entries], [e[3] for e in entries], [e[4] for e in entries],
                                     [e[2] for e in entries], DT)
            else:
                for e in entries:
                    e[0].step(e[3], e[4], None, e[2], DT)
            for e in entries:
                e[3], e[4] = e[4], e[3]
        out = [(e[3].particle_q.clone(), e[3].particle_qd.clone()) for e in entries]
    stream.synchronize()
    return out


@pytest.mark.parametrize("side_stream", [False, True])
def test_batch_equals_steps_in_order(side_stream):
    sizes = (9, 33, 48, 17, 64, 300)  # the last one is beyond the size that runs beside others
    for use in (sizes[:-1], sizes):
        stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
        torch.cuda.synchronize()
        x = _run(_entries(use), 12, True, stream)
        y = _run(_entries(use), 12, False, stream)
        for (qa, va), (qb, vb) in zip(x, y):
            assert torch.equal(qa, qb) and torch.equal(va, vb)


@pytest.mark.parametrize("twice", [False, True])
def test_dependent_entries_run_in_order(twice):
    """One entry's output is the next one's input (and, with ``twice``, both use one solver)."""
    model, q0 = scenes.draped_cloth(n=40, seed=1, height=0.902)
    results = []
    for batch in (True, False):
        s = [SolverVBD(model, iterations=4), SolverVBD(model, iterations=4)]
        if twice:
            s[1] = s[0]
        a, b, c = model.state(), model.state(), model.state()
        a.particle_q.copy_(torch.from_numpy(q0).cuda())
        if batch:
            SolverVBD.step_batch(s, [a, b], [b, c], None, DT)
        else:
            s[0].step(a, b, None, None, DT)
            s[1].step(b, c, None, None, DT)
        torch.cuda.synchronize()
        results.append((c.particle_q.clone(), c.particle_qd.clone()))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


def test_resident_solvers_run_in_order():
    """A resident step takes one CTA per patch on the whole GPU, its patches waiting for one another, so
    two of them never run beside each other."""
    def run(batch):
        entries = []
        for k, n in enumerate((64, 96, 80)):
            model, q0 = scenes.draped_cloth(n=n, seed=k, height=0.902)
            a, b = model.state(), model.state()
            a.particle_q.copy_(torch.from_numpy(q0).cuda())
            pipe = CollisionPipeline(model, soft_contact_margin=5e-3)
            entries.append([SolverVBD(model, iterations=4, resident_step=k < 2), pipe, pipe.contacts(), a, b])
        out = _run(entries, 6, batch, torch.cuda.current_stream())
        for e in entries[:2]:
            assert e[0].step_kernel_info()["resident"] and e[0].status()["timeouts"] == 0
        return out

    for (qa, va), (qb, vb) in zip(run(True), run(False)):
        assert torch.equal(qa, qb) and torch.equal(va, vb)
