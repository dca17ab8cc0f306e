"""The plane step with and without material code (mu, PEC, PMC in every combination) against
the oracle's operator, at sizes on and around the 32 x 8 tile and the plane blocks."""
from __future__ import annotations

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('have', ['', 'mu', 'pec', 'pmc', 'mu pec pmc'])
@pytest.mark.parametrize('shape', [(1, 1, 2), (9, 8, 32), (5, 9, 33), (17, 7, 31), (4, 257, 1)], ids=str)
def test_products_match_the_oracle(cuda, shape, have):
    from meanas_b200.operators import GridOperator
    from meanas_b200.scpml import stretch_all_faces
    from oracle import fdfd_oracle as O
    rng = numpy.random.default_rng(3)
    n = 3 * int(numpy.prod(shape))
    omega = 2 * numpy.pi / 17
    dxes = stretch_all_faces(shape, omega, min([4] + [(s - 1) // 3 for s in shape if s > 1]))
    eps = rng.uniform(1, 12, n)
    mu = rng.uniform(1, 2, n) if 'mu' in have else None
    pec = (rng.random(n) < 0.2).astype(float) if 'pec' in have else None
    pmc = (rng.random(n) < 0.2).astype(float) if 'pmc' in have else None
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    op = GridOperator(omega, dxes, eps, mu, pec, pmc, device=cuda)
    ref = O.e_full_apply(omega, dxes, eps, x, mu, pec, pmc)
    pl = O.precond_pl(dxes)
    sym = pl * O.e_full_apply(omega, dxes, eps, x / pl, mu, pec, pmc)
    sym_h = (pl * O.e_full_apply(omega, dxes, eps, x.conj() / pl, mu, pec, pmc)).conj()
    for name, r in (('A0', ref), ('sym', sym), ('sym_h', sym_h)):
        y = op.apply(x, name).cpu().numpy()
        # some forty roundings of 1.1e-16 (6e-8 in complex64)
        assert numpy.linalg.norm(y - r) <= 5e-15 * numpy.linalg.norm(r), name
        y = op.apply(x, name, 'c64').cpu().numpy()
        assert numpy.linalg.norm(y - r) <= 2.5e-6 * numpy.linalg.norm(r), name


@pytest.mark.parametrize('shape', [(3, 9, 33), (21, 17, 40), (70, 9, 5), (33, 300, 1)], ids=str)
def test_results_do_not_depend_on_the_x_chunk(cuda, shape):
    """The chunk that a plan chooses for itself and any other give the same bits (the passes'
    sums run over a fixed partition)."""
    from meanas_b200.operators import GridOperator
    from meanas_b200.scpml import stretch_all_faces
    rng = numpy.random.default_rng(4)
    n = 3 * int(numpy.prod(shape))
    omega = 2 * numpy.pi / 17
    dxes = stretch_all_faces(shape, omega, min([4] + [(s - 1) // 3 for s in shape if s > 1]))
    op = GridOperator(omega, dxes, rng.uniform(1, 12, n), device=cuda, fp32=False)
    J = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    fields = []
    for chunk in (0, 4, 8, 24, 64):
        op.set_xchunk('c128', chunk)
        E, info = op.solve(J, maxiter=9, rtol=1e-14, criterion='true', profile=True)  # the pass kernels
        fields.append(E.cpu().numpy())
    for f in fields[1:]:
        assert numpy.array_equal(f, fields[0])
