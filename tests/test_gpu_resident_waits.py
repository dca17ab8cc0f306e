"""Resident solves whose waits run out.  ``wait_limit`` sets how many times a CTA reads a word of
another before it gives up; a few reads are fewer than an exchange takes, so CTAs give up at all
points of an iteration, some in an exchange that the others complete."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def problem(cuda):
    from meanas_b200.operators import GridOperator
    from meanas_b200.scpml import stretch_all_faces
    shape = (24, 31, 19)
    n = 3 * int(numpy.prod(shape))
    omega = 2 * numpy.pi / 21 * (1 - 0.25j)
    rng = numpy.random.default_rng(0)
    op = GridOperator(omega, stretch_all_faces(shape, omega.real, 5), numpy.full(n, 2.0), device=cuda)
    return op, rng.standard_normal(n) + 1j * rng.standard_normal(n)


@pytest.mark.parametrize('limit', [1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 64])
@pytest.mark.parametrize('chunk', [1, 2, 0])
@pytest.mark.parametrize('method', ['cocg', 'mixed'])
def test_a_lost_exchange_is_not_taken_for_a_result(problem, method, chunk, limit):
    """The solve ends with an error or with the solution; the next one on the plan is right."""
    from meanas_b200._lib import FDFDError
    op, J = problem
    kw = dict(method=method, rtol=1e-11, criterion='true', chunk=chunk)
    ref, info = op.solve(J, **kw)
    assert info.converged
    for _ in range(4):
        try:
            E, info = op.solve(J, wait_limit=limit, **kw)
        except FDFDError as e:
            assert 'in time' in str(e)
            continue
        # both residuals are at 1e-11; the lossy operator's condition number is below 1e4
        assert info.converged and info.residual <= 1.01e-11
        assert float((E - ref).norm()) <= 1e-7 * float(ref.norm())
    again, _ = op.solve(J, **kw)
    assert numpy.array_equal(again.cpu().numpy(), ref.cpu().numpy())


def test_a_converged_field_has_no_stale_brick(problem):
    """Short solves of one launch per iteration, where other CTAs than the first give up in
    the exchange in which the first one sees the tolerance met."""
    from meanas_b200._lib import FDFDError
    op, J = problem
    _, info = op.solve(J, rtol=1e-11, criterion='true', maxiter=4, record_history=True)
    for rtol in 1.0001 * info.history[1:4]:
        for limit in range(1, 25):
            for _ in range(20):
                try:
                    _, info = op.solve(J, rtol=rtol, criterion='true', chunk=1, wait_limit=limit)
                except FDFDError as e:
                    assert 'in time' in str(e)
                    continue
                # the residual is formed again from the field at the end
                assert info.converged and info.residual <= 1.0001 * rtol, limit


@pytest.mark.parametrize('limit', [-1, -2, -3, -20, 1, 3, 5, 10, 20])
@pytest.mark.parametrize('chunk', [1, 3, 0])
@pytest.mark.parametrize('method,adjoint', [('cocg', False), ('cocg', True), ('mixed', False)])
def test_the_solve_goes_on_without_the_resident_form(problem, method, adjoint, chunk, limit):
    """A wait that runs out, or no (further) resident launch: no error, the same solution, the
    cap on the iterations and a history without gaps."""
    op, J = problem
    kw = dict(method=method, rtol=1e-11, criterion='true', chunk=chunk, adjoint=adjoint, maxiter=4000)
    ref, _ = op.solve(J, **kw)
    for _ in range(3):
        E, info = op.solve(J, wait_limit=limit, record_history=method == 'cocg', **kw)
        assert info.converged and info.residual <= 1.01e-11 and info.iterations <= 4000
        assert float((E - ref).norm()) <= 1e-7 * float(ref.norm())
        if method == 'cocg':
            assert numpy.all(info.history[1:] > 0) and info.history[-1] <= 1e-11
    again, _ = op.solve(J, **kw)
    assert numpy.array_equal(again.cpu().numpy(), ref.cpu().numpy())


@pytest.mark.parametrize('limit', [0, -1, -4, 2, 6])
def test_the_cap_holds_when_the_form_changes(problem, limit):
    op, J = problem
    E, info = op.solve(J, rtol=1e-13, criterion='true', chunk=1, maxiter=7, wait_limit=limit)
    assert (info.status, info.iterations) == ('maxiter', 7)
    assert abs(op.residual(E, J)['rel'] / info.residual - 1) <= 1e-9


def test_chunks_are_cut_to_what_the_counters_hold(cuda):
    """A launch counts CTAs times iterations in 32 bits: a chunk of 2^31 - 1 is cut, with the same
    bits as the default.  (A count that runs over takes 29 million iterations.)"""
    from meanas_b200.operators import GridOperator
    shape = (3, 5, 4)
    n = 3 * int(numpy.prod(shape))
    rng = numpy.random.default_rng(3)
    dxes = [[numpy.ones(m, dtype=complex) for m in shape] for _ in range(2)]
    op = GridOperator(0.5, dxes, numpy.ones(n), device=cuda)
    J = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    kw = dict(rtol=1e-9, criterion='true')
    E, info = op.solve(J, **kw)
    big, ibig = op.solve(J, chunk=2 ** 31 - 1, **kw)
    assert info.converged and ibig.iterations == info.iterations
    assert numpy.array_equal(big.cpu().numpy(), E.cpu().numpy())
