"""The workloads whose speed is tracked, and the same computations in plain torch.

Every case is a dict of plain values with a ``kind``:

* ``solve``    a solve on a kept operator (parameter sweeps, optimisation loops)
* ``stretch``  32 iterations of a long solve, from an earlier field (the iterates of the
               complex-symmetric iteration differ between two roundings from some hundred
               iterations on, so a longer stretch has no value of its own)
* ``refill``   a kept operator loaded with the next problem of its size, then solved (what a
               serving slot does for every request)
* ``generic``  the drop-in ``generic()`` call from host arrays to a host field
* ``grad``     the differentiable solve: forward, loss on a monitor plane, backward
* ``apply``    a matrix-free operator product
* ``post``     E -> H and the Poynting product after a solve
* ``source``   the boundary source before a solve
* ``fdtd``     a run of time steps with a point source
* ``csr``      the assembled-matrix solver behind the ``matrix_solver`` hook

Grids are the shapes of the benchmark, serving and test problems or lie between them.
Permittivities are random axis-aligned blocks in [1, 12.1], cell widths carry SC-PML
layers.  ``q`` is the bandwidth of a solve: ``omega = 2 pi / wavelength (1 - i / (2 q))``,
the complex frequency whose solution is the response averaged over that bandwidth; ``q = 0``
is a real frequency.  Solves run to 1e-12 so that what they return is the solution and not
the iterate at which they happened to stop.
"""
from __future__ import annotations

import math

import numpy
import torch

DEV = 'cuda'
STRETCH = 32     # iterations of a stretch
CAP = 20000      # iterations that no solve here needs


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest request of a serving stream: a 2D grid, where launches and latency count
        dict(name='refill_2d_128', kind='refill', X=128, Y=128, Z=1, pml=10, wavelength=24.0, q=2,
             method='mixed', adjoint=False, masks=False),
        # the smallest 3D request, complex128
        dict(name='solve_3d_32', kind='solve', X=32, Y=32, Z=32, pml=8, wavelength=20.0, q=3,
             method='cocg', adjoint=False, masks=False),
        # the drop-in call on the reference's own size: everything a first-time caller pays
        dict(name='generic_3d_48', kind='generic', X=48, Y=48, Z=48, pml=10, wavelength=30.0, q=0,
             method='cocg', adjoint=False, masks=False),
        # an inverse-design step: forward and adjoint solve and the permittivity gradient
        dict(name='grad_48x48x40', kind='grad', X=48, Y=48, Z=40, pml=8, wavelength=26.0, q=3,
             method='cocg', adjoint=False, masks=False),
        # mixed precision on the largest 3D serving size
        dict(name='solve_mixed_3d_128', kind='solve', X=128, Y=128, Z=128, pml=10, wavelength=24.0, q=2,
             method='mixed', adjoint=False, masks=False),
        # a stretch of the benchmark's long complex128 solve, from an earlier field
        dict(name='stretch_3d_160', kind='stretch', X=160, Y=160, Z=128, pml=12, wavelength=24.0, q=0,
             method='cocg', adjoint=False, masks=False),
        # the same for an adjoint solve with mu and conductors on a ragged grid
        dict(name='stretch_masked_adj_121', kind='stretch', X=121, Y=97, Z=109, pml=10, wavelength=20.0, q=0,
             method='cocg', adjoint=True, masks=True),
        # one product on the benchmark grid: the inner operation of a caller's own Krylov method
        dict(name='apply_c128_160', kind='apply', X=160, Y=160, Z=128, pml=12, op='A0', precision='c128',
             masks=False),
        # fields after a solve, odd sizes
        dict(name='post_121x97x109', kind='post', X=121, Y=97, Z=109, pml=10, masks=True),
        # time stepping: a small float64 run without PML (launches), and the benchmark grid in
        # float32 with CPML on every face
        dict(name='fdtd_f64_40', kind='fdtd', X=40, Y=40, Z=40, steps=40, dtype='float64', cpml=0),
        dict(name='fdtd_f32_cpml_160', kind='fdtd', X=160, Y=160, Z=128, steps=20, dtype='float32', cpml=8),
        # the reference's assembled-matrix flow on the GPU
        dict(name='csr_40x36x32', kind='csr', X=40, Y=36, Z=32, pml=8, wavelength=24.0, q=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, most):
    """Three sizes spread over [lo, hi] on a logarithmic scale, odd ones among them."""
    while True:
        s = [_log_int(rng, lo, hi) for _ in range(3)]
        if s[0] * s[1] * s[2] <= most:
            return s


def draw(rng):
    kind = rng.choice(['solve', 'solve', 'stretch', 'stretch', 'refill', 'generic', 'grad', 'apply', 'apply', 'post',
                       'source', 'fdtd', 'fdtd', 'csr'])
    if kind == 'fdtd':
        big = rng.random() < 0.5
        X, Y, Z = _grid(rng, 24, 160, 160 * 160 * 128) if big else _grid(rng, 20, 64, 64 ** 3)
        if rng.random() < 0.2:
            X, Y, Z = _log_int(rng, 128, 1024), _log_int(rng, 128, 1024), 1
        return dict(kind=kind, X=X, Y=Y, Z=Z, steps=rng.randint(10, 20 if big else 40),
                    dtype=rng.choice(['float32', 'float64']),
                    cpml=0 if Z == 1 else rng.choice([0, 4, 8]))
    if kind in ('apply', 'post', 'source'):
        X, Y, Z = _grid(rng, 24, 176, 160 * 160 * 128)
        if kind == 'apply' and rng.random() < 0.2:
            X, Y, Z = _log_int(rng, 128, 1024), _log_int(rng, 128, 1024), 1
        c = dict(kind=kind, X=X, Y=Y, Z=Z, pml=rng.randint(6, 10), masks=kind != 'source' and rng.random() < 0.4)
        if kind == 'apply':
            c['op'] = rng.choice(['A0', 'A0', 'sym', 'sym_h'])
            c['precision'] = rng.choice(['c128', 'c64'])
        return c
    wavelength = round(rng.uniform(16.0, 40.0), 3)
    if kind == 'csr':
        X, Y, Z = _grid(rng, 24, 48, 40 * 36 * 32)
        return dict(kind=kind, X=X, Y=Y, Z=Z, pml=rng.randint(6, 8), wavelength=wavelength, q=2)
    two_d = kind in ('solve', 'stretch', 'refill') and rng.random() < 0.3
    if kind == 'stretch':
        X, Y, Z = _grid(rng, 32, 200, 160 * 160 * 128)
        if two_d:
            X, Y, Z = _log_int(rng, 128, 1024), _log_int(rng, 128, 1024), 1
    elif two_d:
        X, Y, Z = _log_int(rng, 64, 256), _log_int(rng, 64, 256), 1
    else:
        X, Y, Z = _grid(rng, 28, 80, 64 ** 3)
    method = rng.choice(['cocg', 'mixed']) if kind in ('solve', 'refill') else 'cocg'
    return dict(kind=kind, X=X, Y=Y, Z=Z, pml=rng.randint(8, 10), wavelength=wavelength,
                q=0 if kind == 'stretch' else rng.choice([2, 3]), method=method,
                adjoint=kind in ('solve', 'stretch') and rng.random() < 0.3,
                masks=kind == 'stretch' and rng.random() < 0.3)


# ----------------------------------------------------------------------------- problems
def _shape(case):
    return (int(case['X']), int(case['Y']), int(case['Z']))


def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _blocks(shape, side, lo, hi, fill, g):
    """(3, X, Y, Z): 1, and values in [lo, hi] on random boxes of about ``side`` cells."""
    coarse = [max(1, -(-n // side)) for n in shape]
    v = lo + (hi - lo) * torch.rand(3, *coarse, device=DEV, generator=g, dtype=torch.float64)
    m = torch.rand(1, *coarse, device=DEV, generator=g) < fill
    v = torch.where(m, v, torch.ones_like(v))
    for a, n in enumerate(shape):
        v = v.repeat_interleave(side, dim=1 + a).narrow(1 + a, 0, n)
    return v.contiguous()


def _plates(shape, frac, g):
    """(3, X, Y, Z): 1 on random two-cell plates."""
    coarse = [max(1, -(-shape[0] // 2)), max(1, -(-shape[1] // 12)), max(1, -(-shape[2] // 12))]
    m = (torch.rand(3, *coarse, device=DEV, generator=g) < frac).double()
    for a, (n, side) in enumerate(zip(shape, (2, 12, 12))):
        m = m.repeat_interleave(side, dim=1 + a).narrow(1 + a, 0, n)
    return m.contiguous()


def _widths(shape, omega, thickness):
    """dxes of a unit grid with an SC-PML (polynomial m = 3.5, ln R = -16) on every face
    of every axis longer than one cell."""
    out = [[], []]
    for n in shape:
        i = numpy.arange(n, dtype=float)
        pair = []
        for pos in (i + 0.5, i):
            w = numpy.ones(n, dtype=complex)
            if n > 1 and thickness:
                t = float(thickness)
                s = 1j * (4.5 * -16 / 2) / t / omega.real
                lo = ((t - pos) / t).clip(0, None) * (i < thickness)
                hi = ((pos - (n - t)) / t).clip(0, None) * (i >= n - thickness)
                w = w * (1 + s * lo ** 3.5) * (1 + s * hi ** 3.5)
            pair.append(w)
        out[0].append(pair[0])
        out[1].append(pair[1])
    return out


def _omega(case):
    w = 2 * math.pi / float(case.get('wavelength', 24.0))
    q = case.get('q', 0)
    return complex(w, -w / (2 * q)) if q else complex(w, 0.0)


def _problem(case, seed):
    shape = _shape(case)
    g = _gen(seed)
    omega = _omega(case)
    p = dict(shape=shape, omega=omega, dxes=_widths(shape, omega, case['pml']), mu=None, pec=None, pmc=None)
    if case['kind'] == 'generic':  # a slab core along x, as in the reference's dipole problem
        p['epsilon'] = torch.ones(3, *shape, device=DEV, dtype=torch.float64)
        y, z = shape[1] // 2, shape[2] // 2
        p['epsilon'][:, :, y - 5:y + 5, z - 2:z + 2] = 12.1
    else:
        p['epsilon'] = _blocks(shape, max(4, min(20, max(shape) // 8)), 1.0, 12.1, 0.3, g)
    if case.get('masks'):
        p['mu'] = _blocks(shape, 9, 1.0, 1.5, 0.15, g)
        p['pec'] = _plates(shape, 0.04, g)
        p['pmc'] = _plates(shape, 0.02, g)
    # a Gaussian patch of current (random polarisation and place) near the middle
    at = [n // 2 if n < 8 else n // 2 + int(torch.randint(-(n // 8), n // 8 + 1, (1,), device=DEV, generator=g))
          for n in shape]
    pol = torch.randn(3, device=DEV, generator=g, dtype=torch.complex128)
    r = [torch.exp(-(torch.arange(n, device=DEV, dtype=torch.float64) - c) ** 2 / 8.0) for n, c in zip(shape, at)]
    r = [torch.where(v > 1e-3, v, torch.zeros_like(v)) for v in r]
    J = pol[:, None, None, None] * (r[0][:, None, None] * r[1][:, None] * r[2])
    if p['pec'] is not None:
        J = J * (p['pec'] == 0)
    p['J'] = J.contiguous()
    return p


def _field(shape, seed, salt, dtype=torch.complex128):
    return torch.randn(3, *shape, device=DEV, generator=_gen(seed, salt), dtype=dtype)


def _earlier(shape, seed):
    """A field that fades out towards the PML, as an iterate does."""
    E = _field(shape, seed, 9)
    for a, n in enumerate(shape):
        if n > 1:
            w = torch.sin(math.pi * (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n) ** 2
            E = E * _ax(w, a)
    return E.contiguous()


def _vec(t):
    return None if t is None else t.reshape(-1)


# ----------------------------------------------------------------------------- what a program keeps
def prepare(case, seed):
    kind = case['kind']
    if kind == 'fdtd':
        return _prepare_fdtd(case, seed)
    if kind == 'csr':
        from meanas_b200.csr import CsrMatrix
        p = _problem(dict(case, masks=False), seed)
        data, cols, indptr, b = _symmetrised_csr(p)
        M = CsrMatrix((data.cpu().numpy(), cols.cpu().numpy(), indptr.cpu().numpy()), DEV)
        return dict(case=case, M=M, b=b)
    from meanas_b200.operators import GridOperator
    if kind in ('apply', 'post', 'source'):
        p = _problem(case, seed)
        x = _field(p['shape'], seed, 5,
                   torch.complex64 if case.get('precision') == 'c64' else torch.complex128).reshape(-1)
        st = dict(case=case, x=x)
        if kind == 'source':
            from meanas_b200 import fields
            st['op'] = fields.e_boundary_source(_vec(_region(p['shape'])), p['omega'], p['dxes'], _vec(p['epsilon']),
                                                device=DEV)
        else:
            st['op'] = GridOperator(p['omega'], p['dxes'], _vec(p['epsilon']), _vec(p['mu']), _vec(p['pec']),
                                    _vec(p['pmc']), device=DEV, fp32=case.get('precision') == 'c64')
        return st
    p = _problem(case, seed)
    st = dict(case=case, p={k: (_vec(v) if isinstance(v, torch.Tensor) else v) for k, v in p.items()})
    if kind == 'generic':
        st['p'] = {k: (v.cpu().numpy() if isinstance(v, torch.Tensor) else v) for k, v in st['p'].items()}
    elif kind == 'grad':
        m = torch.zeros(3, *p['shape'], device=DEV)
        m[:, (3 * p['shape'][0]) // 4] = 1.0
        st['monitor'] = m.reshape(-1)
        st['eps'] = st['p']['epsilon'].clone().requires_grad_(True)
    else:
        q = st['p']
        st['op'] = GridOperator(q['omega'], q['dxes'], q['epsilon'].clone(), q['mu'], q['pec'], q['pmc'], device=DEV,
                                fp32=case['method'] == 'mixed')
        st['E'] = torch.empty_like(q['J'])
        if kind == 'stretch':
            st['guess'] = _earlier(p['shape'], seed).reshape(-1)
    return st


def _prepare_fdtd(case, seed):
    from meanas_b200 import fdtd
    shape = _shape(case)
    dt_ = torch.float32 if case['dtype'] == 'float32' else torch.float64
    e, h, eps = _fdtd_fields(case, seed)
    dxes = _fdtd_widths(shape)
    st = dict(case=case, e=e.to(dt_), h=h.to(dt_), eps=eps)
    if case['cpml']:
        par = [[None if n == 1 else fdtd.cpml_params(axis=a, polarity=pol, dt=0.5, thickness=case['cpml'],
                                                     epsilon_eff=1.5, cfs_alpha=0.05)
                for pol in (-1, 1)] for a, n in enumerate(shape)]
        ue, uh = fdtd.updates_with_cpml(par, 0.5, dxes, eps, device=DEV)
        st['step_h'], st['step_e'] = (lambda: uh(st['e'], st['h'])), (lambda: ue(st['e'], st['h']))
    else:
        mh, me = fdtd.maxwell_h(0.5, dxes, device=DEV), fdtd.maxwell_e(0.5, dxes, device=DEV)
        st['step_h'], st['step_e'] = (lambda: mh(st['e'], st['h'])), (lambda: me(st['e'], st['h'], eps))
    st['probe'] = st['e'][(2, *(n // 2 for n in shape))]
    st['pulse'] = [_pulse(t) for t in range(case['steps'])]
    return st


def _pulse(t):
    return math.sin(0.35 * t) * math.exp(-((t - 12) / 6) ** 2)


def _fdtd_widths(shape):
    """Real widths, mildly graded along x."""
    return [[1.0 + (0.1 * numpy.sin(numpy.arange(n) / 7.0) if a == 0 else numpy.zeros(n))
             for a, n in enumerate(shape)] for _ in range(2)]


def _fdtd_fields(case, seed):
    shape = _shape(case)
    g = _gen(seed, 7)
    e = torch.randn(3, *shape, device=DEV, generator=g, dtype=torch.float32)
    h = torch.randn(3, *shape, device=DEV, generator=g, dtype=torch.float32)
    return e, h, _blocks(shape, 12, 1.0, 12.1, 0.3, g)


# ----------------------------------------------------------------------------- one pass
def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'solve':
        E, _ = state['op'].solve(state['p']['J'], method=case['method'], rtol=1e-12, criterion='true',
                                 adjoint=case['adjoint'], maxiter=CAP)
        return E
    if kind == 'stretch':
        E, _ = state['op'].solve(state['p']['J'], E_guess=state['guess'], method=case['method'], rtol=1e-12,
                                 criterion='true', adjoint=case['adjoint'], maxiter=STRETCH)
        return E
    if kind == 'refill':
        p = state['p']
        state['op'].update(p['omega'], p['dxes'], p['epsilon'], p['mu'], p['pec'], p['pmc'])
        E, _ = state['op'].solve(p['J'], out=state['E'], method=case['method'], rtol=1e-12, criterion='true',
                                 maxiter=CAP)
        return E
    if kind == 'generic':
        from meanas_b200 import generic
        p = state['p']
        return generic(p['omega'], p['dxes'], p['J'], p['epsilon'], p['mu'], pec=p['pec'], pmc=p['pmc'],
                       matrix_solver_opts=dict(rtol=1e-12, maxiter=CAP), criterion='true', device=DEV)
    if kind == 'grad':
        from meanas_b200.autograd import fdfd_solve
        p, eps = state['p'], state['eps']
        eps.grad = None
        E = fdfd_solve(eps, p['J'], p['omega'], p['dxes'], rtol=1e-12, maxiter=CAP)
        ((E.real ** 2 + E.imag ** 2) * state['monitor']).sum().backward()
        return E.detach(), eps.grad
    if kind == 'apply':
        return state['op'].apply(state['x'], case['op'], case['precision'])
    if kind == 'post':
        return state['op'].poynting(state['x'])
    if kind == 'source':
        return state['op'] @ state['x']
    if kind == 'fdtd':
        for v in state['pulse']:
            state['step_h']()
            state['step_e']()
            state['probe'] += v
        return state['e'], state['h']
    x, _ = state['M'].solve(state['b'], rtol=1e-12, maxiter=CAP)
    return x


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: inputs and outputs once; for an iterative solve, every iteration reads and
    writes the iterate, the residual and the direction once and reads the permittivity, for
    the usual number of iterations to 1e-12 at this bandwidth."""
    n = case['X'] * case['Y'] * case['Z']
    kind = case['kind']
    if kind == 'fdtd':
        b = 4 if case['dtype'] == 'float32' else 8
        # a step reads and writes both fields and reads epsilon; eight operations and a division a component
        return dict(bytes=case['steps'] * n * (3 * 4 * b + 24), flops=case['steps'] * n * 60)
    if kind == 'apply':
        b = 16 if case['precision'] == 'c128' else 8
        extra = (3 * b // 2 + 1) if case['masks'] else 0
        return dict(bytes=n * (6 * b + 3 * b // 2 + extra), flops=n * 170)
    if kind == 'post':
        return dict(bytes=n * (144 + (25 if case['masks'] else 0)), flops=n * 150)
    if kind == 'source':
        return dict(bytes=n * (96 + 24 + 24), flops=n * 340)
    its = _iterations(case)
    if kind == 'csr':
        nnz, rows = 39 * n, 3 * n
        return dict(bytes=its * 2 * (20 * nnz + 6 * 16 * rows), flops=its * 2 * 8 * nnz)
    extra = 25 if case['masks'] else 0
    if case['method'] == 'mixed':
        return dict(bytes=its * n * (6 * 24 + 12 + extra), flops=its * n * 450)
    solves = 2 if kind == 'grad' else 1
    return dict(bytes=solves * its * n * (6 * 48 + 24 + extra), flops=solves * its * n * 260)


def _iterations(case):
    if case['kind'] == 'stretch':
        return STRETCH
    return 1600 if case['q'] in (0, 2) else 2200


# ----------------------------------------------------------------------------- the same in plain torch, 64 bits
def _ax(w, a):
    s = [1, 1, 1]
    s[a] = -1
    return w.reshape(s)


def _tab(dxes):
    return [[_ax(torch.as_tensor(numpy.asarray(w, dtype=complex), device=DEV), a) for a, w in enumerate(side)]
            for side in dxes]


def _curl(f, w, sign):
    """Forward (sign = -1) or backward (sign = 1) curl of a (3, X, Y, Z) field."""
    def d(c, a):
        diff = torch.roll(f[c], sign, dims=a) - f[c]
        return (diff if sign < 0 else -diff) / w[a]
    return torch.stack([d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)])


def _free(m):
    return None if m is None else (m == 0).to(torch.float64)


def _product(p):
    """x -> A0 x and the weights W = p^2 for a problem of _problem()."""
    e, h = _tab(p['dxes'])
    pe, pm = _free(p['pec']), _free(p['pmc'])
    w2 = p['omega'] ** 2

    def A0(x):
        x = x if pe is None else x * pe
        f = _curl(x, e, -1)
        f = f if p['mu'] is None else f / p['mu']
        f = f if pm is None else f * pm
        y = _curl(f, h, 1) - w2 * p['epsilon'] * x
        return y if pe is None else y * pe
    W = torch.stack([(e[0] * h[1] * h[2]).expand(p['shape']), (h[0] * e[1] * h[2]).expand(p['shape']),
                     (h[0] * h[1] * e[2]).expand(p['shape'])])
    return A0, W


def _cocg(A0, W, b, tol=1e-13, most=20000):
    """Conjugate gradients for the form sum(u W v), in which A0 is symmetric; restarted from
    the true residual until that is small."""
    x, bn = torch.zeros_like(b), b.norm()
    for _ in range(3):
        r = b - A0(x)
        if r.norm() <= tol * bn:
            break
        p, rho = r.clone(), (r * W * r).sum()
        for k in range(most):
            q = A0(p)
            a = rho / (p * W * q).sum()
            x = x + a * p
            r = r - a * q
            if k % 25 == 24 and r.norm() <= tol * bn:
                break
            rho, old = (r * W * r).sum(), rho
            p = r + (rho / old) * p
    return x


def _cocg_steps(A0, W, b, x, steps):
    """The iterate after so many steps from x."""
    r = b - A0(x)
    p, rho = r.clone(), (r * W * r).sum()
    for _ in range(steps):
        q = A0(p)
        a = rho / (p * W * q).sum()
        x = x + a * p
        r = r - a * q
        rho, old = (r * W * r).sum(), rho
        p = r + (rho / old) * p
    return x


def _solved(p, b0, adjoint=False, guess=None, steps=None):
    A0, W = _product(p)
    pe = _free(p['pec'])
    b = b0 if pe is None else b0 * pe

    def solver(b, x):
        return _cocg(A0, W, b) if steps is None else _cocg_steps(A0, W, b, x, steps)
    if not adjoint:
        return solver(b, guess)
    # A0^H E = b in the variable y of E = conj(W y)
    return (W * solver(b.conj() / W, None if guess is None else guess.conj() / W)).conj().resolve_conj()


def _region(shape):
    """A total-field box in the middle of the grid."""
    q = torch.zeros(3, *shape, device=DEV, dtype=torch.float64)
    q[:, shape[0] // 4:3 * shape[0] // 4, shape[1] // 4:3 * shape[1] // 4,
      shape[2] // 4:max(1, 3 * shape[2] // 4)] = 1.0
    return q


def exact(case, seed):
    kind = case['kind']
    if kind == 'fdtd':
        return _fdtd_exact(case, seed)
    n = case['X'] * case['Y'] * case['Z']
    p = _problem(dict(case, masks=False) if kind == 'csr' else case, seed)
    if kind == 'apply':
        A0, W = _product(p)
        x = _field(p['shape'], seed, 5, torch.complex64 if case['precision'] == 'c64' else torch.complex128)
        x = x.to(torch.complex128)
        if case['op'] == 'A0':
            return A0(x).reshape(-1)
        pl = torch.sqrt(W)
        y = pl * A0(x / pl) if case['op'] == 'sym' else (pl * A0(x.conj() / pl)).conj().resolve_conj()
        return y.reshape(-1)
    if kind == 'post':
        e, h = _tab(p['dxes'])
        E = _field(p['shape'], seed, 5)
        H = _curl(E, e, -1)
        H = H if p['mu'] is None else H / p['mu']
        H = H if p['pmc'] is None else H * _free(p['pmc'])
        H = H / (-1j * p['omega'])
        ew = [E[a] * e[a] for a in range(3)]
        hw = [H[a].conj() * h[a] for a in range(3)]
        S = torch.stack([torch.roll(ew[(a + 1) % 3], -1, a) * hw[(a + 2) % 3]
                         - torch.roll(ew[(a + 2) % 3], -1, a) * hw[(a + 1) % 3] for a in range(3)])
        return S.reshape(-1), H.reshape(-1)
    if kind == 'source':
        A0, _ = _product(p)
        E, Q = _field(p['shape'], seed, 5), _region(p['shape'])
        J = (A0(Q * E) - Q * A0(E)) / (-1j * p['omega'])
        edge = torch.zeros_like(Q, dtype=torch.bool)
        for a in range(1, 4):
            if Q.shape[a] > 1:
                m = Q.shape[a]
                for idx in (list(range(1, m)) + [m - 1], [0] + list(range(m - 1))):
                    edge |= Q.index_select(a, torch.tensor(idx, device=DEV)) != Q
        return (J * edge).reshape(-1)
    # solves: plain conjugate gradients; None where that takes too long
    if n * (_iterations(case) + 200) * (2 if kind == 'grad' else 1) > 8e9:
        return None
    b0 = -1j * p['omega'] * p['J']
    if kind == 'csr':
        _, W = _product(p)
        return (torch.sqrt(W) * _solved(p, b0)).reshape(-1)
    if kind == 'stretch':
        return _solved(p, b0, case['adjoint'], _earlier(p['shape'], seed), STRETCH).reshape(-1)
    E = _solved(p, b0, bool(case.get('adjoint')))
    if kind == 'grad':
        m = torch.zeros_like(E)
        m[:, (3 * p['shape'][0]) // 4] = 1.0
        Ea = _solved(p, 2 * E * m, True)
        return E.reshape(-1), (p['omega'] ** 2 * Ea.conj() * E).real.reshape(-1)
    return E.reshape(-1)


def _symmetrised_csr(p):
    """(data, columns, row pointers, b) of Pl A0 Pr x = Pl b0, built from index arithmetic."""
    shape, N = p['shape'], p['shape'][0] * p['shape'][1] * p['shape'][2]
    e, h = _tab(p['dxes'])
    ids = torch.arange(N, device=DEV).reshape(shape)
    rows, cols, vals = [], [], []

    def terms(c, sign):
        """The four terms (component, axis shift, coefficient) of a curl's component c."""
        u, v = (c + 1) % 3, (c + 2) % 3
        for comp, a, s in ((v, u, 1.0), (u, v, -1.0)):
            w = (e if sign < 0 else h)[a].expand(shape)
            yield comp, a, sign, (s if sign < 0 else -s) / w
            yield comp, a, 0, (-s if sign < 0 else s) / w
    for c in range(3):
        for hc, a1, s1, w1 in terms(c, 1):
            at1 = torch.roll(ids, s1, a1) if s1 else ids
            for ec, a2, s2, w2 in terms(hc, -1):
                at2 = torch.roll(ids, s2, a2) if s2 else ids
                rows.append((c * N + ids).reshape(-1))
                cols.append((ec * N + at2.reshape(-1)[at1.reshape(-1)]).reshape(-1))
                vals.append((w1.reshape(-1) * w2.reshape(-1)[at1.reshape(-1)]))
        rows.append((c * N + ids).reshape(-1))
        cols.append((c * N + ids).reshape(-1))
        vals.append((-p['omega'] ** 2 * p['epsilon'][c]).reshape(-1).to(torch.complex128))
    rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    _, W = _product(p)
    pl = torch.sqrt(W).reshape(-1)
    vals = pl[rows] * vals / pl[cols]
    key, inv = torch.unique(rows * (3 * N) + cols, return_inverse=True)
    data = torch.zeros(key.numel(), dtype=torch.complex128, device=DEV)
    torch.view_as_real(data).index_add_(0, inv, torch.view_as_real(vals))
    indptr = torch.zeros(3 * N + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(key // (3 * N), minlength=3 * N), 0)
    return data, key % (3 * N), indptr, pl * (-1j * p['omega'] * p['J']).reshape(-1)


def _fdtd_exact(case, seed):
    shape, dt = _shape(case), 0.5
    dev_dt = torch.float32 if case['dtype'] == 'float32' else torch.float64
    e, h, eps = _fdtd_fields(case, seed)
    e, h = e.to(dev_dt).double(), h.to(dev_dt).double()
    f, b = ([_ax(torch.as_tensor(w, device=DEV), a) for a, w in enumerate(side)] for side in _fdtd_widths(shape))
    th = case['cpml']
    psi, par = {}, {}
    if th:
        f = b
        sigma_max, kappa_max = 1.6 / 2 * 4.5, math.sqrt(1.5)
        for a, n in enumerate(shape):
            for pp in range(2 if n > 1 else 0):
                for side in (0, 1):  # E, H positions of the layers
                    x = numpy.arange(1, th + 1, dtype=float) - (0.5 if (pp == 1) == (side == 0) else 0.0)
                    x = x if pp else x[::-1]
                    s = (x / th) ** 3.5
                    sg, kp, al = s * sigma_max, 1 + s * (kappa_max - 1), (1 - x / th) * 0.05
                    p0 = numpy.exp(-(sg / kp + al) * dt)
                    par[a, pp, side] = [_ax(torch.as_tensor(numpy.ascontiguousarray(v), device=DEV), a)
                                        for v in (p0, sg / (sg + kp * al) * (p0 - 1), 1 / kp)]
                    z = list(shape)
                    z[a] = th
                    psi[a, pp, side] = [torch.zeros(z, device=DEV, dtype=torch.float64) for _ in range(2)]

    def curl(fld, w, sign, side):
        d = {}
        for a in range(3):
            for c in range(3):
                if c != a:
                    diff = torch.roll(fld[c], sign, dims=a) - fld[c]
                    d[a, c] = (diff if sign < 0 else -diff) / w[a]
        extra = torch.zeros_like(fld)
        for (a, pp, sd), (pu, pv) in psi.items():
            if sd != side:
                continue
            u, v = [c for c in range(3) if c != a]
            se = -1.0 if a != 1 else 1.0
            p0, p1, p2 = par[a, pp, sd]
            at = (0 if pp == 0 else shape[a] - th)
            du, dv, eu, ev = (t.narrow(a, at, th) for t in (d[a, u], d[a, v], extra[u], extra[v]))
            du *= p2
            dv *= p2
            pu.mul_(p0).add_(p1 * dv)
            pv.mul_(p0).add_(p1 * du)
            eu += se * pu
            ev -= se * pv
        out = torch.stack([d[1, 2] - d[2, 1], d[2, 0] - d[0, 2], d[0, 1] - d[1, 0]])
        return out + extra

    for t in range(case['steps']):
        h -= dt * curl(e, f, -1, 1)
        e += dt / eps * curl(h, b, 1, 0)
        e[(2, *(n // 2 for n in shape))] += _pulse(t)
    return e, h
