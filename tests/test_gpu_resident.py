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


MIXED = [(1, 1, 1), (2, 1, 3), (5, 4, 1), (3, 60, 7), (31, 33, 29), (48, 48, 48), (52, 52, 52), (57, 56, 57),
         (128, 128, 1), (389, 380, 1), (410, 410, 1)]


def _shadow(n, seed):
    """The solver's hashed shadow vector (``shadow`` in fdfd_ops.cuh)."""
    def mix(x):
        for shift, mul in ((16, 0x7feb352d), (15, 0x846ca68b), (16, 1)):
            x = (x ^ (x >> numpy.uint32(shift))) * numpy.uint32(mul)
        return x
    with numpy.errstate(over='ignore'):
        a = mix(numpy.arange(n, dtype=numpy.uint32) ^ numpy.uint32(seed))
        b = mix(a ^ numpy.uint32(((seed << 16) | (seed >> 16)) & 0xffffffff) ^ numpy.uint32(0x9e3779b9))
    return (a * 2.0 ** -32 - 0.5) + 1j * (b * 2.0 ** -32 - 0.5)


def _bicgstab(A, b, shadow, steps, dtype):
    """The iterate after ``steps`` of BiCGSTAB from zero, vectors in ``dtype``, sums in FP64."""
    def dot(u, v):
        return complex(numpy.vdot(u.astype(complex), v.astype(complex)))
    A, r, rh = A.astype(dtype), b.astype(dtype), shadow.astype(dtype)
    x, p, rho = numpy.zeros_like(r), r.copy(), dot(rh, r)
    for _ in range(steps):
        v = A @ p
        alpha = rho / dot(rh, v)
        s = r - dtype(alpha) * v
        t = A @ s
        omega = dot(t, s) / dot(t, t).real
        x = x + dtype(alpha) * p + dtype(omega) * s
        r = s - dtype(omega) * t
        rho_new = -omega * dot(rh, t)
        beta = rho_new / rho * alpha / omega
        rho = rho_new
        p = r + dtype(beta) * (p - dtype(omega) * v)
    return x.astype(complex)


@pytest.mark.parametrize('masks', [False, True])
@pytest.mark.parametrize('shape', MIXED, ids=str)
def test_bicgstab_iterates_match_the_oracle(cuda, shape, masks):
    """One and three iterations (the second launch goes on from the first one's state)
    against the same recurrence in complex128 on the host.  How far complex64 takes an
    iterate off depends on the problem, so the host's complex64 iterate sets the scale: ten
    times its error and 1e-6 (sixteen roundings of 6e-8)."""
    from meanas_b200.operators import GridOperator
    from oracle import fdfd_oracle as O
    p, J, _ = _problem(shape, masks, seed=1)
    if numpy.prod(shape) < 8:
        pytest.skip('three steps exhaust the Krylov space')
    op = GridOperator(**p, device=cuda)
    A = O.e_full_csr(p['omega'], p['dxes'], p['epsilon'], p['mu'], p['pec'], p['pmc'])
    b = -1j * p['omega'] * J
    if masks:
        b = numpy.where(p['pec'] > 0, 0, b)
    bn = numpy.linalg.norm(b)
    for steps in (1, 3):
        E, info = op.solve(J, method='mixed', rtol=1e-13, criterion='true', maxiter=steps, max_outer=1,
                           inner_rtol=1e-6, chunk=2)
        E = E.cpu().numpy()
        # the seed of the first refinement step's shadow vector
        ref, single = (bn * _bicgstab(A, b / bn, _shadow(len(b), 0x5eed5eed), steps, t)
                       for t in (numpy.complex128, numpy.complex64))
        assert info.iterations == steps
        size = numpy.linalg.norm(ref)
        scale = numpy.linalg.norm(single - ref) / size
        assert numpy.linalg.norm(E - ref) <= (1e-6 + 10 * scale) * size, (steps, scale)
        E2, _ = op.solve(J, method='mixed', rtol=1e-13, criterion='true', maxiter=steps, max_outer=1,
                         inner_rtol=1e-6, chunk=2)
        assert numpy.array_equal(E2.cpu().numpy(), E)  # fixed order of all sums


@pytest.mark.parametrize('shape', [(24, 31, 19), (100, 90, 1), (40, 40, 40)], ids=str)
def test_mixed_solution_matches_cocg(cuda, shape):
    """Converged to 1e-11, several launches and refinements: the two methods' fields agree."""
    from meanas_b200.operators import GridOperator
    p, J, _ = _problem(shape, False, seed=2)
    p['omega'] = p['omega'] * (1 - 0.25j)
    p['epsilon'][:] = 2.0
    op = GridOperator(**p, device=cuda)
    E, info = op.solve(J, method='mixed', rtol=1e-11, criterion='true', chunk=40)
    Er, ref = op.solve(J, method='cocg', rtol=1e-11, criterion='true')
    assert info.converged and ref.converged and info.residual <= 1e-11 * 1.01
    # both residuals are at 1e-11; the lossy operator's condition number is below 1e4
    assert float((E - Er).norm()) <= 1e-7 * float(Er.norm())


@pytest.mark.parametrize('steps', [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize('shape', [(9, 8, 33), (12, 70, 1)], ids=str)
def test_owed_updates_are_made_wherever_the_loop_stops(cuda, shape, steps):
    """The two-launch form owes its x updates for a pass: after any number of iterations the
    field equals the resident form's, which makes them at once (few steps: only the order
    of the sums differs, 1e-16 times a cancellation below 1e3)."""
    from meanas_b200.operators import GridOperator
    p, J, guess = _problem(shape, False, seed=3)
    op = GridOperator(**p, device=cuda, fp32=False)
    kw = dict(rtol=1e-13, criterion='true', maxiter=steps, E_guess=guess)
    E, info = op.solve(J, **kw)
    Er, ref = op.solve(J, profile=True, **kw)
    assert info.iterations == ref.iterations == steps
    assert float((E - Er).norm()) <= 1e-12 * float(Er.norm())


@pytest.mark.parametrize('steps', [1, 2, 3, 4, 5])
def test_updates_two_at_a_time(cuda, steps):
    """From a million cells on, x is updated in every second pass; an all-zero
    conductor mask selects the update in every pass on the same problem: the same field."""
    from meanas_b200.operators import GridOperator
    p, J, _ = _problem((129, 64, 128), False, seed=3)
    J = numpy.where(numpy.arange(J.size) % 977 == 500, J, 0)
    op = GridOperator(**p, device=cuda, fp32=False)
    E, info = op.solve(J, rtol=1e-13, criterion='true', maxiter=steps)
    p['pmc'] = numpy.zeros(J.size)
    ref_op = GridOperator(**p, device=cuda, fp32=False)
    Er, ref = ref_op.solve(J, rtol=1e-13, criterion='true', maxiter=steps)
    assert info.iterations == ref.iterations == steps
    assert float((E - Er).norm()) <= 1e-13 * float(Er.norm())
