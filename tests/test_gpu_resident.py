"""Resident solves (grids held on the SMs by one cooperative launch) against the two-launch
form of the same iteration, which ``profile=True`` selects: single cells and planes, axes
shorter than a brick, ragged bricks, one and two cells per thread, the largest grids that fit
and the first that do not, flat grids, materials and conductors, adjoint solves.

Both forms run the same recurrences and differ in the order of their sums only, so after 16
iterations the iterates agree to the rounding of the sums (1e-16) times the cancellation of
the unconjugated forms (at most 1e4 this early) and a few: 1e-10 leaves a margin."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu

COCG = [(1, 1, 1), (2, 1, 3), (5, 4, 1), (1, 40, 1), (3, 60, 7), (16, 15, 17), (31, 33, 29), (48, 48, 48), (52, 52, 52),
        (54, 54, 54), (200, 13, 11), (128, 128, 1), (381, 379, 1), (400, 400, 1)]


def _problem(shape, masks, seed=0):
    from meanas_b200.scpml import stretch_all_faces
    rng = numpy.random.default_rng(seed)
    omega = 2 * numpy.pi / 21
    pml = min([6] + [(n - 1) // 3 for n in shape if n > 1])
    dxes = stretch_all_faces(shape, omega, pml)
    n = 3 * int(numpy.prod(shape))
    p = dict(omega=omega, dxes=dxes, epsilon=rng.uniform(1, 12, n), mu=None, pec=None, pmc=None)
    if masks:
        p['mu'] = rng.uniform(1, 1.5, n)
        p['pec'] = (rng.random(n) < 0.05).astype(float)
        p['pmc'] = (rng.random(n) < 0.03).astype(float)
    J = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    guess = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return p, J, guess


@pytest.mark.parametrize('masks,adjoint', [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize('shape', COCG, ids=str)
def test_cocg_iterates_match_the_two_launch_form(cuda, shape, masks, adjoint):
    from meanas_b200.operators import GridOperator
    p, J, guess = _problem(shape, masks)
    op = GridOperator(**p, device=cuda, fp32=False)
    kw = dict(rtol=1e-13, criterion='true', adjoint=adjoint, maxiter=16, chunk=7, E_guess=guess, record_history=True)
    E, info = op.solve(J, **kw)
    Er, ref = op.solve(J, profile=True, **kw)
    E, Er = E.cpu().numpy(), Er.cpu().numpy()
    assert (info.status, info.iterations) == (ref.status, ref.iterations)
    assert numpy.linalg.norm(E - Er) <= 1e-10 * numpy.linalg.norm(Er)
    assert numpy.allclose(info.history, ref.history, rtol=1e-6, atol=1e-12)
    E2, _ = op.solve(J, **kw)  # fixed order of all sums: the same bits again
    assert numpy.array_equal(E2.cpu().numpy(), E)
