"""FDTD half steps bit for bit against the oracle where the kernel branches: flat grids, axes of
one cell, layers that fill or overlap an axis, width tables too long for shared memory, and
values and widths at and beyond the range of the tabled-reciprocal division."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    a, b = numpy.asarray(a), numpy.asarray(b)
    return numpy.array_equal(numpy.isnan(a), numpy.isnan(b)) and \
        numpy.array_equal(a.view(a.dtype.str.replace('f', 'i'))[~numpy.isnan(a)],
                          b.view(b.dtype.str.replace('f', 'i'))[~numpy.isnan(b)])


def _fields(shape, dtype, rng, special):
    e, h = (rng.standard_normal((3, *shape)) * 10.0 ** rng.uniform(-12, 3, (3, *shape)) for _ in range(2))
    if special:
        tiny = numpy.finfo(dtype).tiny
        pick = numpy.array([0.0, -0.0, tiny, -tiny / 4, numpy.finfo(dtype).max, numpy.inf, -numpy.inf, numpy.nan])
        for f in (e, h):
            m = rng.random(f.shape) < 0.05
            f[m] = rng.choice(pick, int(m.sum()))
            f[rng.random(f.shape) < 0.2] = 0.0
    return e.astype(dtype), h.astype(dtype)


@pytest.mark.parametrize('special', [False, True], ids=['plain', 'special'])
@pytest.mark.parametrize('dtype', ['float32', 'float64'])
@pytest.mark.parametrize('shape', [(1, 1, 1), (7, 1, 1), (1, 9, 33), (300, 31, 1), (6, 5, 4), (13, 17, 257), (2040, 3, 9)],
                         ids=str)
def test_plain_steps(cuda, shape, dtype, special):
    import torch
    from meanas_b200 import fdtd
    from oracle import fdfd_oracle as O
    rng = numpy.random.default_rng(4)
    dx = [[rng.choice([1.0, 0.7, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 3.1e-9], n) for n in shape] for _ in range(2)]
    if special:
        dx[0][0][0], dx[1][-1][-1] = 1e-200, 5e-324
    eps = rng.choice([1.0, 2.1, 12.1], (3, *shape))
    e, h = _fields(shape, dtype, rng, special)
    et, ht = torch.as_tensor(e, device=cuda), torch.as_tensor(h, device=cuda)
    mh, me = fdtd.maxwell_h(0.4, dx, device=cuda), fdtd.maxwell_e(0.4, dx, device=cuda)
    with numpy.errstate(all='ignore'):
        for _ in range(3):
            mh(et, ht)
            me(et, ht, eps)
            # the curls of the reference are arrays of the field type
            h -= 0.4 * O.curl_forward(dx[0], e)
            e += 0.4 * O.curl_back(dx[1], h) / eps
    assert _same(et.cpu().numpy(), e) and _same(ht.cpu().numpy(), h)


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
@pytest.mark.parametrize('psi', ['float32', 'float64'])
@pytest.mark.parametrize('shape,layers', [((12, 11, 10), ((4, 4), (4, 4), (4, 4))), ((9, 8, 34), ((0, 4), (4, 0), (4, 5))),
                                          ((8, 9, 8), ((4, 4), (5, 4), (4, 4))), ((7, 6, 7), ((4, 4), (4, 4), (5, 6))),
                                          ((40, 21, 9), ((5, 0), (0, 0), (9, 0))), ((2050, 5, 7), ((8, 8), (0, 0), (3, 3)))],
                         ids=str)
def test_cpml_steps(cuda, shape, layers, psi, dtype):
    import torch
    from meanas_b200 import fdtd
    from oracle import fdfd_oracle as O
    rng = numpy.random.default_rng(5)
    dx = [[rng.uniform(0.8, 1.3, n) for n in shape] for _ in range(2)]
    eps, mu = rng.choice([1.0, 2.1, 12.1], (3, *shape)), rng.uniform(1, 2, (3, *shape))
    par = [[None, None] for _ in range(3)]
    tab = [[None, None] for _ in range(3)]
    for a in range(3):
        for pp, pol in enumerate((-1, 1)):
            if layers[a][pp]:
                q = fdtd.cpml_params(axis=a, polarity=pol, dt=0.4, thickness=layers[a][pp], epsilon_eff=1.5, cfs_alpha=0.05)
                par[a][pp] = q
                tab[a][pp] = tuple(numpy.stack([numpy.ravel(v) for v in q[s]]) for s in ('param_e', 'param_h'))
    e, h = _fields(shape, dtype, rng, False)
    et, ht = torch.as_tensor(e, device=cuda), torch.as_tensor(h, device=cuda)
    ue, uh = fdtd.updates_with_cpml(par, 0.4, dx, eps, dtype=numpy.dtype(psi), device=cuda)
    ref = O.CpmlUpdates(tab, 0.4, dx, shape, dtype=numpy.dtype(psi))
    for t in range(4):
        uh(et, ht, mu if t % 2 else None)
        ref.update_H(e, h, mu if t % 2 else (1, 1, 1))
        ue(et, ht)
        ref.update_E(e, h, eps)
    assert _same(et.cpu().numpy(), e) and _same(ht.cpu().numpy(), h)
