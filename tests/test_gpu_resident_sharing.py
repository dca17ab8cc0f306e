"""Resident solves by CTAs of half an SM: the sizes at which the split changes, and solves on
several streams at once, among them one that is too large to run resident."""
from __future__ import annotations

import threading

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _problem(shape, masks, seed=0, lossy=False):
    from meanas_b200.scpml import stretch_all_faces
    rng = numpy.random.default_rng(seed)
    omega = 2 * numpy.pi / 21
    dxes = stretch_all_faces(shape, omega, min([6] + [(n - 1) // 3 for n in shape if n > 1]))
    n = 3 * int(numpy.prod(shape))
    p = dict(omega=omega * (1 - 0.25j) if lossy else omega, dxes=dxes,
             epsilon=numpy.full(n, 2.0) if lossy else rng.uniform(1, 12, n), mu=None, pec=None, pmc=None)
    if masks:
        p['mu'] = rng.uniform(1, 1.5, n)
        p['pec'] = (rng.random(n) < 0.05).astype(float)
        p['pmc'] = (rng.random(n) < 0.03).astype(float)
    J, guess = (rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(2))
    return p, J, guess


# 148 CTAs x 256 cells, x 512 cells on flat grids, and one plane more; 256 threads with ragged bricks
EDGES = [(148, 16, 16), (149, 16, 16), (148, 256, 1), (149, 256, 1), (296, 256, 1), (297, 256, 1), (29, 30, 31),
         (251, 261, 1), (36, 36, 36)]


def _iterate(p, J, x, shape, steps, dtype):
    """The field after ``steps`` of COCG from ``x``, in numpy and ``dtype``."""
    def widths(side):
        return [numpy.asarray(w, dtype=dtype).reshape([-1 if a == i else 1 for i in range(3)])
                for a, w in enumerate(p['dxes'][side])]

    def free(name):
        return 1 if p[name] is None else (p[name].reshape(3, *shape) == 0).astype(dtype)

    def curl(f, w, sign):
        def d(c, a):
            diff = numpy.roll(f[c], sign, axis=a) - f[c]
            return (diff if sign < 0 else -diff) / w[a]
        return numpy.stack([d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)])
    e, h = widths(0), widths(1)
    pe, pm = free('pec'), free('pmc')
    mu = 1 if p['mu'] is None else p['mu'].reshape(3, *shape).astype(dtype)
    w2eps = dtype(p['omega']) ** 2 * p['epsilon'].reshape(3, *shape).astype(dtype)

    def A(v):
        v = v * pe
        return (curl(curl(v, e, -1) / mu * pm, h, 1) - w2eps * v) * pe
    W = numpy.stack([numpy.broadcast_to(w, shape) for w in (e[0] * h[1] * h[2], h[0] * e[1] * h[2], h[0] * h[1] * e[2])])
    x = x.reshape(3, *shape).astype(dtype)
    r = dtype(-1j) * dtype(p['omega']) * J.reshape(3, *shape).astype(dtype) * pe - A(x)
    q, rho = r, (r * W * r).sum()
    for _ in range(steps):
        v = A(q)
        alpha = rho / (q * W * v).sum()
        x, r = x + alpha * q, r - alpha * v
        old, rho = rho, (r * W * r).sum()
        q = r + (rho / old) * q
    return x.reshape(-1)


@pytest.mark.parametrize('masks', [False, True])
@pytest.mark.parametrize('shape', EDGES, ids=str)
def test_edges_of_the_split(cuda, shape, masks):
    """COCG after 8 iterations, in launches of 7 and 1, against the host's in 64-bit mantissas.
    How far rounding takes an iterate off depends on the problem (the unconjugated forms
    cancel), so the host's complex128 iterate sets the scale: ten times its error and some
    hundred roundings.  Mixed precision against COCG, converged to 1e-11 with a condition number
    below 1e4."""
    from meanas_b200.operators import GridOperator
    p, J, guess = _problem(shape, masks)
    op = GridOperator(**p, device=cuda, fp32=False)
    E, info = op.solve(J, rtol=1e-13, criterion='true', maxiter=8, chunk=7, E_guess=guess)
    assert info.iterations == 8
    ref, double = (_iterate(p, J, guess, shape, 8, t) for t in (numpy.clongdouble, numpy.complex128))
    size = numpy.linalg.norm(ref.astype(complex))
    scale = numpy.linalg.norm((double - ref).astype(complex)) / size
    assert numpy.linalg.norm((E.cpu().numpy() - ref).astype(complex)) <= (1e-14 + 10 * scale) * size
    p, J, _ = _problem(shape, masks, lossy=True)
    op = GridOperator(**p, device=cuda)
    if masks:
        J = numpy.where(p['pec'] > 0, 0, J)
    E, info = op.solve(J, method='mixed', rtol=1e-11, criterion='true', chunk=40)
    Er, ref = op.solve(J, method='cocg', rtol=1e-11, criterion='true')
    assert info.converged and ref.converged and info.residual <= 1.01e-11
    assert float((E - Er).norm()) <= 1e-7 * float(Er.norm())


def test_solves_at_once_give_the_same_bits(cuda):
    import torch
    from meanas_b200.operators import GridOperator
    jobs = []
    for k, (shape, method, masks, maxiter) in enumerate([
            ((32, 32, 32), 'cocg', False, 700), ((128, 128, 1), 'mixed', False, 900), ((64, 60, 58), 'cocg', False, 300),
            ((24, 25, 23), 'cocg', True, 700), ((48, 48, 48), 'mixed', False, 400), ((128, 128, 1), 'cocg', False, 900),
            ((250, 255, 1), 'mixed', True, 600), ((66, 57, 61), 'mixed', False, 300)]):
        p, J, _ = _problem(shape, masks, seed=k)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            op = GridOperator(**p, device=cuda)
        jobs.append((op, torch.as_tensor(J, device=cuda), s, dict(method=method, rtol=1e-12, criterion='true', maxiter=maxiter)))

    def solve(k, out):
        op, J, s, kw = jobs[k]
        with torch.cuda.stream(s):
            out[k] = op.solve(J, **kw)[0].cpu().numpy()
    torch.cuda.synchronize()
    alone, together = {}, {}
    for k in range(len(jobs)):
        solve(k, alone)
    for _ in range(2):
        threads = [threading.Thread(target=solve, args=(k, together)) for k in range(len(jobs))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(len(jobs)):
            assert numpy.array_equal(alone[k], together[k]), k


@pytest.mark.parametrize('method', ['cocg', 'mixed'])
@pytest.mark.parametrize('shape,most', [((40, 40, 40), 64), ((30, 30, 30), 256)], ids=str)
def test_whole_sm_launches_are_short(cuda, shape, method, most):
    """Launches that have the GPU to themselves end after 64 iterations, so that kernels of other
    streams get their turn; the result does not depend on it."""
    from meanas_b200.operators import GridOperator
    p, J, _ = _problem(shape, False)
    op = GridOperator(**p, device=cuda)
    kw = dict(method=method, rtol=1e-13, criterion='true', maxiter=512, max_outer=1, inner_rtol=1e-12)
    E, info = op.solve(J, **kw)
    # two launches are under way when a solve ends, and about ten kernels come before and after
    assert 512 // most <= info.kernel_launches <= 512 // most + 15
    other, _ = op.solve(J, chunk=100, **kw)
    assert numpy.array_equal(other.cpu().numpy(), E.cpu().numpy())
