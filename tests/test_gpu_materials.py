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
