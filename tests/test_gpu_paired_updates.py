"""COCG's paired x updates (grids of 2^20 cells and more without mu and conductors) where the loop
stops with an update owed: after a discarded step, inside the stencil pass, at the cap; on flat
and 3D grids.  Unit cells, periodic, eps = 1: Ez that varies along x and y only has plane waves as
eigenvectors, so the breakdowns can be set and the iterates are known."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1024, 1024, 1), (128, 64, 128)]
OMEGA2 = 0.05


def _operator(cuda, shape, omega, pmc=None):
    from meanas_b200.operators import GridOperator
    dxes = [[numpy.ones(n, dtype=complex) for n in shape] for _ in range(2)]
    op = GridOperator(omega, dxes, numpy.ones(3 * int(numpy.prod(shape))), pmc=pmc, device=cuda, fp32=False)
    assert not op.resident('cocg')
    return op


def _pair(cuda, shape, omega):
    """The paired form and, by a conductor mask of zeros, the form that updates x in every pass."""
    return _operator(cuda, shape, omega), _operator(cuda, shape, omega, numpy.zeros(3 * int(numpy.prod(shape))))


def _ez(shape, field):
    out = numpy.zeros((3, *shape), dtype=complex)
    out[2] = field
    return out.ravel()


def _weights(lam):
    """Weights of eigenvalues ``lam`` (the last one chosen) for which p^T A p of step
    len(lam) - 2 (from 0) vanishes: the Hankel determinant of the moments 1, 2, ... is zero,
    and it is affine in every weight."""
    s = len(lam) - 1

    def det(last):
        w = numpy.array([1.0] * s + [last], dtype=numpy.longdouble)
        m = [(w * lam ** k).sum() for k in range(2 * s + 1)]
        h = [[m[i + j + 1] for j in range(s)] for i in range(s)]

        def minor(a):
            return a[0][0] if len(a) == 1 else sum((-1) ** c * a[0][c] * minor([r[:c] + r[c + 1:] for r in a[1:]])
                                                   for c in range(len(a)))
        return minor(h)
    d0, d1 = det(0), det(1)
    return numpy.array([1.0] * s + [-d0 / (d1 - d0)], dtype=numpy.longdouble)


@pytest.mark.parametrize('steps', [1, 2, 3])
@pytest.mark.parametrize('shape', SHAPES, ids=str)
def test_a_discarded_step_leaves_the_field_before_it(cuda, shape, steps):
    """p^T A p of step ``steps`` is zero but for rounding: the residual explodes, the step is
    discarded and, at the cap, the field is the iterate before it, whichever of its updates
    are owed.  (A few steps from well separated eigenvalues: sums that cancel by less than
    1e4, so 1e-10.)"""
    freq = numpy.array([1 / 16, 3 / 16, 5 / 16, 7 / 16, 1 / 2][:steps + 2])
    lam = 4 * numpy.sin(numpy.pi * freq.astype(numpy.longdouble)) ** 2 - OMEGA2
    w = _weights(lam)
    norm = numpy.where(freq == 0.5, 1.0, 0.5)  # of cos^2 per cell
    amp = numpy.sqrt((w / norm).astype(numpy.clongdouble))
    # the recurrence on the amplitudes
    r, x = amp.copy(), 0 * amp
    p, rho = r, (w + 0 * r).sum()
    for _ in range(steps):
        alpha = rho / (norm * lam * p * p).sum()
        x, r = x + alpha * p, r - alpha * lam * p
        rho, old = (norm * r * r).sum(), rho
        p = r + rho / old * p
    waves = numpy.cos(2 * numpy.pi * freq[:, None] * numpy.arange(shape[0]))
    omega = numpy.sqrt(OMEGA2)

    def along_x(a):
        return _ez(shape, (a.astype(complex)[:, None] * waves).sum(0)[:, None, None])
    op = _operator(cuda, shape, omega)
    E, info = op.solve(along_x(amp) / (-1j * omega), rtol=1e-13, criterion='true', maxiter=steps + 1)
    assert (info.status, info.iterations) == ('maxiter', steps + 1)
    want = along_x(x)
    assert numpy.linalg.norm(E.cpu().numpy() - want) <= 1e-10 * numpy.linalg.norm(want)


@pytest.mark.parametrize('maxiter', [2, 3, 4])
@pytest.mark.parametrize('shape', SHAPES, ids=str)
def test_a_stop_inside_the_stencil_pass(cuda, shape, maxiter):
    """Integer fields and eigenvalues -1, 1, 3 with weights 1, 3, -1: alpha = -3, beta = -16 and
    p^T A p = 0 exactly in the second pass, which has one update owed.  The restart goes on
    from x = -3 b (an update lost or made twice is an error of its size) and both forms take the
    same steps from there, up to rounding and what the restarted forms cancel (1e4)."""
    X, Y, _ = shape
    i, j = numpy.arange(X)[:, None, None], numpy.arange(Y)[None, :, None]
    two = numpy.array([1, 1, -1, -1])
    b = 1 + two[i % 4] + two[(i + 1) % 4] + two[j % 4] + 1j * numpy.where(i % 2, -1, 1)
    J = _ez(shape, 1j * b)  # -i omega J = b
    paired, single = _pair(cuda, shape, 1.0)
    kw = dict(rtol=1e-13, criterion='true', maxiter=maxiter)
    E, info = paired.solve(J, **kw)
    Es, infos = single.solve(J, **kw)
    assert (info.status, info.iterations) == (infos.status, infos.iterations) == ('maxiter', maxiter)
    assert float((E - Es).norm()) <= 1e-10 * float(Es.norm())


@pytest.mark.parametrize('steps', [1, 2, 3, 4, 5])
@pytest.mark.parametrize('shape', SHAPES, ids=str)
def test_updates_owed_at_the_cap_from_a_guess(cuda, shape, steps):
    """Real right-hand side and guess: r^T W r does not cancel and few eigenvalues are
    negative, so five steps amplify roundings of 1e-16 by less than 1e3."""
    rng = numpy.random.default_rng(6)
    n = 3 * int(numpy.prod(shape))
    J, guess = 1j * rng.standard_normal(n), rng.standard_normal(n)
    paired, single = _pair(cuda, shape, numpy.sqrt(OMEGA2))
    kw = dict(rtol=1e-13, criterion='true', maxiter=steps, E_guess=guess)
    E, info = paired.solve(J, **kw)
    Es, infos = single.solve(J, **kw)
    assert info.iterations == infos.iterations == steps
    assert float((E - Es).norm()) <= 1e-13 * float(Es.norm())
