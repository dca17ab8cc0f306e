"""Serving slots on both sides of the resident limit: slots of small grids time no x chunk; a slot
of a larger one replays its captured graphs on problem after problem."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _serve(cuda, precision, shape, count):
    from meanas_b200 import serving, workloads
    rng = numpy.random.default_rng(7)
    probs = [workloads.serving_request(rng, shape=shape) for _ in range(count)]
    with serving.FDFDServer(cuda, max_active=1, precision=precision, rtol=1e-8) as srv:
        res = [srv.submit(serving.Request(p.omega, p.dxes, p.J, p.epsilon)).result() for p in probs]
        return probs, res, dict(srv.stats)


@pytest.mark.parametrize('precision', ['mixed', 'fp64'])
def test_resident_slots_time_no_chunk(cuda, precision):
    from meanas_b200 import operators
    _, res, stats = _serve(cuda, precision, (47, 52, 1), 2)
    assert all(r.info.converged for r in res)
    assert stats['slot_new'] == 1 and stats['slot_tuned'] == 0 and stats['slot_reuse'] == 1
    assert not [k for k in operators._TUNED if k[1] == (47, 52, 1)]


@pytest.mark.parametrize('precision', ['mixed', 'fp64'])
def test_graphs_are_replayed_on_refilled_plans(cuda, precision):
    """The second and third request of a slot: same bits as on a plan of their own (which
    captures its graphs anew), and the oracle's residual."""
    from meanas_b200.operators import GridOperator
    from oracle import fdfd_oracle as O
    shape, method = (60, 57, 62), 'mixed' if precision == 'mixed' else 'cocg'
    probs, res, stats = _serve(cuda, precision, shape, 3)
    assert stats['slot_new'] == 1 and stats['slot_tuned'] == 1 and stats['slot_reuse'] == 2
    for p, r in zip(probs, res):
        assert r.info.converged and O.true_residual(p.omega, p.dxes, p.epsilon, r.E, p.J) <= 1.01e-8
        op = GridOperator(p.omega, p.dxes, p.epsilon, device=cuda, fp32=precision == 'mixed')
        assert not op.resident(method)
        E, _ = op.solve(p.J, method=method, rtol=1e-8, criterion='true', maxiter=200000)
        assert numpy.array_equal(E.cpu().numpy(), r.E)
