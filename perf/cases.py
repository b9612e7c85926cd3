"""Performance cases of the finite-difference path.

A case is one call (or one fixed group of calls) that a program using this
package makes over and over: a band-batched stencil, the fused
pseudo-Hamiltonian, the band preconditioner, a grid transfer, a Poisson solve.
Sizes follow the workloads of bench.py and the tests; draw() spreads them over
the ranges that such programs use.  exact() restates every call in 64-bit
torch operations.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from gpaw_b200.density import interpolate_pseudo_density
from gpaw_b200.fd_operators import Gradient, Laplace, apply_pseudo_hamiltonian
from gpaw_b200.grid_descriptor import GridDescriptor
from gpaw_b200.poisson import PoissonSolver
from gpaw_b200.preconditioner import Preconditioner
from gpaw_b200.serving import PoissonBatch
from gpaw_b200.transformers import Transformer

BOHR = 0.52917721092
DTYPES = {'float64': torch.float64, 'float32': torch.float32,
          'complex128': torch.complex128, 'complex64': torch.complex64}
ITEM = {'float64': 8, 'float32': 4, 'complex128': 16, 'complex64': 8}
EPS = 2e-10


def listed():
    return [
        # A small molecule: 16 real bands in a box with zero boundaries, one
        # kinetic apply.  A call of tens of microseconds.
        dict(name='laplace_f64_box', kind='laplace', dtype='float64', n0=48, n1=48, n2=48,
             pbc=False, nn=3, bands=16, k=0.0),
        # A bulk cell with a k-point: the kinetic operator on 512 complex bands.
        dict(name='laplace_c128_bulk', kind='laplace', dtype='complex128', n0=96, n1=96, n2=96,
             pbc=True, nn=3, bands=512, k=0.25),
        # Gradients along all three axes (stress, currents, dipoles) in the
        # single-precision variant, on a slab-like grid of unequal sides.
        dict(name='gradient_c64_slab', kind='gradient', dtype='complex64', n0=120, n1=64, n2=80,
             pbc=True, nn=3, bands=64, k=0.25),
        # The eigensolver's H psi: kinetic operator plus local potential, on a
        # ragged grid.
        dict(name='hamiltonian_c128', kind='hamiltonian', dtype='complex128', n0=84, n1=90,
             n2=100, pbc=True, nn=3, bands=64, k=0.125),
        # A primitive fcc cell (non-orthogonal, six stencil directions) with
        # a k-point.
        dict(name='laplace_c128_fcc', kind='skew', cell='fcc', dtype='complex128', n0=48, n1=48,
             n2=48, pbc=True, nn=3, bands=96, k=0.25),
        # One preconditioner call of the eigensolver on a block of bands.
        dict(name='precondition_c128', kind='precondition', dtype='complex128', n0=96, n1=96,
             n2=96, pbc=True, nn=3, bands=64, k=0.25),
        # Fine to coarse grid (nn = 3), many arrays at once: the largest data.
        dict(name='restrict_f64', kind='restrict', dtype='float64', n0=112, n1=112, n2=112,
             pbc=True, nn=3, bands=256),
        # Coarse to fine grid.
        dict(name='interpolate_f64', kind='interpolate', dtype='float64', n0=112, n1=112, n2=112,
             pbc=True, nn=3, bands=64),
        # Every SCF step: the pseudo density of two spins to the fine grid of a
        # zero-boundary cell, renormalised.
        dict(name='density_f64', kind='density', dtype='float64', n0=64, n1=64, n2=72, pbc=False,
             nn=3, bands=2),
        # Every SCF step: one Poisson solve, plain and in mixed precision.
        dict(name='poisson_f64', kind='poisson', n0=128, n1=128, n2=128, pbc=False, nn=3,
             relax='J', precision='fp64', charges=64),
        dict(name='poisson_mixed', kind='poisson', n0=128, n1=128, n2=128, pbc=False, nn=3,
             relax='J', precision='mixed', charges=64),
        # Pair densities: 32 independent solves on grids of four sizes, one
        # graph launch.
        dict(name='poisson_batch_gs', kind='batch', sizes='48,64,80,96', each=8, nn=3,
             relax='GS', precision='fp64', charges=16),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, lo, hi, step=1):
    """Three grid sizes of one case: a common length scale, sides within 30%."""
    base = _log(rng, lo, hi)
    return [max(lo, min(hi, int(round(base * rng.uniform(0.8, 1.2) / step)) * step))
            for _ in range(3)]


def draw(rng):
    kind = rng.choice(['laplace', 'laplace', 'gradient', 'hamiltonian', 'skew', 'precondition',
                       'restrict', 'interpolate', 'density', 'poisson', 'poisson', 'batch'])
    k = rng.choice([0.0, 0.125, 0.25, 0.5])
    if kind in ('laplace', 'gradient', 'hamiltonian'):
        dtype = rng.choice(['float64', 'float32', 'complex128', 'complex128', 'complex64'])
        n = _grid(rng, 24, 144)
        most = 2.0e8 * 8 / ITEM[dtype] / (n[0] * n[1] * n[2])
        return dict(kind=kind, dtype=dtype, n0=n[0], n1=n[1], n2=n[2],
                    pbc=rng.random() < 0.6, nn=rng.choice([2, 3, 3, 3, 4]),
                    bands=max(1, int(_log(rng, 1, max(2, min(512, most))))), k=k)
    if kind == 'skew':
        cell = rng.choice(['fcc', 'bcc', 'hex'])
        n = int(_log(rng, 16, 80))
        dtype = rng.choice(['float64', 'complex128', 'complex128'])
        most = 1.0e8 * 8 / ITEM[dtype] / n ** 3
        return dict(kind=kind, cell=cell, dtype=dtype, n0=n, n1=n, n2=n, pbc=True,
                    nn=rng.choice([2, 3, 3]),
                    bands=max(1, int(_log(rng, 1, max(2, min(256, most))))), k=k)
    if kind == 'precondition':
        dtype = rng.choice(['float64', 'complex128', 'complex128'])
        n = _grid(rng, 24, 112, 4)
        most = 1.0e8 * 8 / ITEM[dtype] / (n[0] * n[1] * n[2])
        return dict(kind=kind, dtype=dtype, n0=n[0], n1=n[1], n2=n[2], pbc=rng.random() < 0.6,
                    nn=3, bands=max(1, int(_log(rng, 1, max(2, min(128, most))))), k=k)
    if kind in ('restrict', 'interpolate'):
        dtype = rng.choice(['float64', 'float64', 'float32', 'complex128'])
        n = _grid(rng, 20, 120)
        most = 1.0e9 / ITEM[dtype] / (n[0] * n[1] * n[2])
        return dict(kind=kind, dtype=dtype, n0=n[0], n1=n[1], n2=n[2], pbc=rng.random() < 0.6,
                    nn=rng.choice([1, 2, 3, 3, 3]),
                    bands=max(1, int(_log(rng, 1, max(2, min(256, most))))))
    if kind == 'density':
        n = _grid(rng, 24, 120)
        return dict(kind=kind, dtype='float64', n0=n[0], n1=n[1], n2=n[2],
                    pbc=rng.random() < 0.4, nn=3, bands=rng.choice([1, 2]))
    if kind == 'poisson':
        n = _grid(rng, 32, 160, 8)
        return dict(kind=kind, n0=n[0], n1=n[1], n2=n[2], pbc=rng.random() < 0.4, nn=3,
                    relax=rng.choice(['J', 'J', 'GS']),
                    precision=rng.choice(['fp64', 'mixed']), charges=rng.randint(8, 64))
    sizes = rng.sample([32, 40, 48, 56, 64, 80, 96], rng.randint(1, 4))
    return dict(kind='batch', sizes=','.join(str(s) for s in sizes), each=rng.randint(2, 8), nn=3,
                relax=rng.choice(['J', 'GS']), precision='fp64', charges=16)


# -- inputs ------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return g


def _n(case):
    return case['n0'], case['n1'], case['n2']


def _cell(case, h=0.18 / BOHR):
    """Lattice vectors (rows) with a grid spacing of about h."""
    n = np.array(_n(case), float)
    if case.get('cell') == 'fcc':
        return np.array([[0, 1, 1], [1, 0, 1], [1, 1, 0]]) * h * n[0] / math.sqrt(2.0)
    if case.get('cell') == 'bcc':
        return np.array([[-1, 1, 1], [1, -1, 1], [1, 1, -1]]) * h * n[0] / math.sqrt(3.0)
    if case.get('cell') == 'hex':
        return np.array([[1, 0, 0], [-0.5, math.sqrt(0.75), 0], [0, 0, 0.9]]) * h * n[0]
    return np.diag(h * n)


def _phases(case):
    """Bloch phases of the k-point (k, 0, 0) in reduced units, or None."""
    if not case['dtype'].startswith('complex'):
        return None
    k_c = np.array([case['k'], 0.0, 0.0])
    sdisp_cd = np.array([[1, -1]] * 3) if case['pbc'] else np.zeros((3, 2), int)
    return np.exp(2j * math.pi * sdisp_cd * k_c[:, None])


def _bands(gd, case, seed):
    """Bands of independent normal values (wave functions, residuals)."""
    dtype = DTYPES[case['dtype']]
    shape = (case['bands'],) + tuple(int(x) for x in gd.n_c)
    return torch.randn(shape, dtype=dtype, device='cuda', generator=_gen(seed))


def _gaussians(gd, n, seed, width=(0.4, 1.2), wall=2.0):
    """A neutral pseudo charge density: n normalised Gaussians of charge +-1
    (widths in Angstrom), their centres at least `wall` from the walls."""
    rng = np.random.RandomState(seed % (1 << 31))
    L = gd.cell_cv.diagonal()
    wall = np.minimum(wall / BOHR, 0.3 * L)
    axes = [torch.arange(int(b), int(e), device='cuda', dtype=torch.float64) * h
            for b, e, h in zip(gd.beg_c, gd.end_c, gd.h_cv.diagonal())]
    rho = torch.zeros(tuple(int(x) for x in gd.n_c), dtype=torch.float64, device='cuda')
    sign = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    for i in range(n):
        s = rng.uniform(*width) / BOHR
        c = rng.uniform(wall, L - wall)
        e = []
        for x, c0, length, periodic in zip(axes, c, L, gd.pbc_c):
            d = x - c0
            if periodic:
                d = d - length * torch.round(d / length)
            e.append(torch.exp(-d * d / (2 * s * s)))
        g = e[0][:, None, None] * e[1][:, None] * e[2]
        rho += g * (sign[i] / (g.sum() * gd.dv))
    return rho - rho.mean()


def _gd(case, h=0.18 / BOHR):
    return GridDescriptor(_n(case), _cell(case, h), case['pbc'])


def _batch_sizes(case):
    return [int(s) for s in case['sizes'].split(',')] * case['each']


def prepare(case, seed):
    kind = case['kind']
    s = SimpleNamespace(kind=kind)
    if kind in ('laplace', 'gradient', 'hamiltonian', 'skew'):
        gd = _gd(case)
        dtype = DTYPES[case['dtype']]
        s.phases = _phases(case)
        s.x = _bands(gd, case, seed)
        if kind == 'gradient':
            s.ops = [Gradient(gd, v, 1.0, case['nn'], dtype) for v in range(3)]
        else:
            s.ops = [Laplace(gd, -0.5, case['nn'], dtype)]
        s.out = [torch.empty_like(s.x) for _ in s.ops]
        if kind == 'hamiltonian':
            real = torch.float32 if case['dtype'] in ('float32', 'complex64') else torch.float64
            s.vt = torch.randn(tuple(int(x) for x in gd.n_c), dtype=real, device='cuda',
                               generator=_gen(seed + 1))
    elif kind == 'precondition':
        gd = _gd(case)
        dtype = DTYPES[case['dtype']]
        s.x = _bands(gd, case, seed)
        s.kpt = SimpleNamespace(phase_cd=_phases(case))
        s.pc = Preconditioner(gd, Laplace(gd, -0.5, case['nn'], dtype), dtype, case['bands'])
    elif kind in ('restrict', 'interpolate', 'density'):
        coarse = _gd(case, 0.2 / BOHR)
        fine = coarse.refine()
        a, b = (fine, coarse) if kind == 'restrict' else (coarse, fine)
        dtype = DTYPES[case['dtype']]
        s.tr = Transformer(a, b, case['nn'], dtype)
        s.x = _bands(a, case, seed)
        s.y = b.empty((case['bands'],), dtype)
        if kind == 'density':
            s.x = s.x.abs_()
            s.fine = fine
            s.charge = _charge(case)
    elif kind == 'poisson':
        gd = _gd(case, 0.2 / BOHR)
        s.solver = PoissonSolver(case['nn'], case['relax'], EPS, case['precision'])
        s.solver.set_grid_descriptor(gd)
        s.solver.prepare()
        s.rho = _gaussians(gd, case['charges'], seed)
        s.phi = gd.empty()
    else:
        s.rhos, s.phis, solvers = [], [], []
        for i, n in enumerate(_batch_sizes(case)):
            gd = GridDescriptor((n,) * 3, (n * 0.2 / BOHR,) * 3, False)
            solver = PoissonSolver(case['nn'], case['relax'], EPS, case['precision'])
            solver.set_grid_descriptor(gd)
            solvers.append(solver)
            s.rhos.append(_gaussians(gd, case['charges'], 1000 * seed + i))
            s.phis.append(gd.empty())
        s.batch = PoissonBatch(solvers)
    return s


def _charge(case):
    return 10.0 * case['bands']


# -- one pass ----------------------------------------------------------------
def run(s):
    if s.kind in ('laplace', 'gradient', 'skew'):
        for op, out in zip(s.ops, s.out):
            op.apply(s.x, out, s.phases)
        return s.out
    if s.kind == 'hamiltonian':
        apply_pseudo_hamiltonian(s.ops[0], s.x, s.out[0], s.vt, s.phases)
        return s.out
    if s.kind == 'precondition':
        return s.pc(s.x, s.kpt)
    if s.kind in ('restrict', 'interpolate'):
        s.tr.apply(s.x, s.y)
        return s.y
    if s.kind == 'density':
        return interpolate_pseudo_density(s.tr, s.x, s.y, s.fine, s.charge)
    if s.kind == 'poisson':
        s.phi.zero_()
        niter = s.solver.solve(s.phi, s.rho)
        return {'phi': s.phi, 'niter': niter}
    for phi in s.phis:
        phi.zero_()
    got = s.batch.solve(s.phis, s.rhos, EPS)
    return {'phi': s.phis, 'niter': [g[0] for g in got]}


# -- what a pass cannot do without --------------------------------------------
def _points(n, pbc):
    return math.prod(x if pbc else x - 1 for x in n)


def _solve_work(n, pbc, precision):
    """One Poisson solve: rho and the guess in, phi out, and per V-cycle (the
    solves take about 12) the level-0 sweeps, residuals and transfers as one
    read of each operand and one write of each result."""
    p = _points(n, pbc)
    cycles = 12
    coarse = 8.0 / 7.0 - 1.0
    # level 0: 3 sweeps (24 B), residual to res (24), norm (16), correction
    # (16), restriction (8); each coarser level 8 sweeps and the same passes.
    cycle = 3 * 24 + 24 + 16 + 16 + 8 + coarse * (8 * 24 + 24 + 16 + 8)
    if precision == 'mixed':
        cycle = 0.5 * cycle + 24 + 20 + 12
    flops = cycles * p * (5 * 39 + coarse * 9 * 15 + 20)
    return {'bytes': float(24 * p + cycles * cycle * p), 'flops': float(flops)}


def work(case):
    kind = case['kind']
    if kind == 'batch':
        w = [_solve_work((n, n, n), False, case['precision']) for n in _batch_sizes(case)]
        return {k: sum(x[k] for x in w) for k in ('bytes', 'flops')}
    if kind == 'poisson':
        return _solve_work(_n(case), case['pbc'], case['precision'])
    p = _points(_n(case), case['pbc'])
    item = ITEM[case['dtype']]
    parts = 2 if case['dtype'].startswith('complex') else 1
    pts = p * case['bands']
    nn = case['nn']
    if kind in ('laplace', 'hamiltonian'):
        extra = p * item / parts if kind == 'hamiltonian' else 0
        return {'bytes': float(2 * item * pts + extra),
                'flops': float(pts * parts * 2 * (6 * nn + 1))}
    if kind == 'gradient':
        return {'bytes': float(4 * item * pts), 'flops': float(3 * pts * parts * 4 * nn)}
    if kind == 'skew':
        dirs = {'fcc': 6, 'bcc': 4, 'hex': 4}[case['cell']]
        return {'bytes': float(2 * item * pts), 'flops': float(pts * parts * 2 * (2 * dirs * nn + 1))}
    if kind == 'precondition':
        # R in, result out; the coarse levels' arrays in between are small.
        return {'bytes': float(2 * item * pts * (1 + 1 / 8.0)),
                'flops': float(pts * parts * (2 * (6 * nn + 1) + 30))}
    fine = _points([2 * x for x in _n(case)], case['pbc']) * case['bands']
    taps = 2 * nn
    per = {'restrict': 2 * (taps + 1) * (1 / 2 + 1 / 4 + 1 / 8),
           'interpolate': 2 * taps * (1 / 2 + 1 / 4 + 1 / 8) / 2,
           'density': 2 * taps * (1 / 2 + 1 / 4 + 1 / 8) / 2 + 2}[kind]
    return {'bytes': float(item * (pts + fine)), 'flops': float(fine * parts * per)}


def tolerance(case):
    """Four times what exact() and the path differ by, measured over listed and
    drawn cases: sums in another order give 2e-16 to 4e-16 in 64 bits (the
    skew stencils' solved weights 1e-15, the gradient's inverted ones 1e-14)
    and 5e-8 to 8e-8 in 32 bits; a Poisson solve stops at the same V-cycle and
    carries the rounding of its sweeps, 1e-15 to 6e-14 (mixed form, 32-bit
    sweeps: 1e-10)."""
    kind = case['kind']
    if kind in ('poisson', 'batch'):
        if case['precision'] == 'mixed':
            return {'rel': 5e-10, 'max': 2e-9}
        return {'rel': 2.5e-13, 'max': 2.5e-12}
    if case['dtype'] in ('float32', 'complex64'):
        return {'rel': 4e-7, 'max': 4e-6}
    if kind == 'gradient':
        return {'rel': 4e-14, 'max': 4e-13}
    if kind == 'skew':
        return {'rel': 4e-15, 'max': 4e-14}
    return {'rel': 2e-15, 'max': 2e-14}


# -- the same in 64-bit torch ---------------------------------------------------
def _second(nn):
    """Central second-difference weights of distance 0..nn, order 2 nn."""
    w = [0.0] + [2.0 * (-1) ** (m + 1) * math.factorial(nn) ** 2 /
                 (m * m * math.factorial(nn - m) * math.factorial(nn + m))
                 for m in range(1, nn + 1)]
    w[0] = -2.0 * sum(w[1:])
    return w


def _first(nn):
    """Central first-difference weights of distance 1..nn."""
    return [(-1) ** (m + 1) * math.factorial(nn) ** 2 /
            (m * math.factorial(nn - m) * math.factorial(nn + m)) for m in range(1, nn + 1)]


def _laplace_terms(case, n, scale, nn, h=0.18 / BOHR):
    """[(offset, weight)] of scale * nabla^2 on the case's cell."""
    w = _second(nn)
    cell = case.get('cell')
    e = np.eye(3, dtype=int)
    if cell == 'fcc':
        dirs = [(d, 0.5) for d in (e[0], e[1], e[2], e[0] - e[1], e[0] - e[2], e[1] - e[2])]
    elif cell == 'bcc':
        dirs = [(d, 0.75) for d in (e[0], e[1], e[2], e[0] + e[1] + e[2])]
    elif cell == 'hex':
        dirs = [(d, 2.0 / 3.0) for d in (e[0], e[1], e[0] + e[1])] + [(e[2], 1 / 0.81)]
    else:
        dirs = [(d, 1.0) for d in e]
    a = scale / h ** 2
    terms = [((0, 0, 0), a * w[0] * sum(x for _, x in dirs))]
    for d, x in dirs:
        for m in range(1, nn + 1):
            terms += [(tuple(m * d), a * x * w[m]), (tuple(-m * d), a * x * w[m])]
    return terms


def _halo(a, width, pbc, phases=None):
    """a (bands, n0, n1, n2) with `width` more points on every side: zeros, or
    the periodic images times the Bloch phases."""
    for ax in range(3):
        d = ax + 1
        n = a.shape[d]
        if pbc:
            lo, hi = a.narrow(d, n - width, width), a.narrow(d, 0, width)
            if phases is not None:
                lo, hi = lo * complex(phases[ax][1]), hi * complex(phases[ax][0])
        else:
            shape = list(a.shape)
            shape[d] = width
            lo = hi = torch.zeros(shape, dtype=a.dtype, device=a.device)
        a = torch.cat((lo, a, hi), d)
    return a


def _stencil(a, terms, pbc, phases=None):
    width = max(max(abs(x) for x in o) for o, _ in terms)
    p = _halo(a, width, pbc, phases)
    out = torch.zeros_like(a)
    for o, w in terms:
        out += w * p[(slice(None),) + tuple(slice(width + int(x), width + int(x) + n)
                                            for x, n in zip(o, a.shape[1:]))]
    return out


def _midpoint(nn):
    """Lagrange weights of the 2 nn points around a midpoint, by distance."""
    x = [2 * i + 1 for i in range(-nn, nn)]
    return [math.prod(-xj / (x[nn + m] - xj) for xj in x if xj != x[nn + m]) for m in range(nn)]


def _restrict(a, nn, pbc, phases=None):
    w = _midpoint(nn)
    W = 2 * nn - 1
    p = _halo(a, W, pbc, phases)
    for d in (1, 2, 3):
        n = a.shape[d]
        c0, m = (0, n // 2) if pbc else (1, (n - 1) // 2)
        take = lambda o: p.narrow(d, W + c0 + o, 2 * m - 1)[(slice(None),) * d + (slice(0, None, 2),)]  # noqa: E731
        q = take(0)
        for j in range(nn):
            q = q + w[j] * (take(2 * j + 1) + take(-2 * j - 1))
        p = 0.5 * q
    return p


def _interpolate(a, nn, pbc, phases=None):
    w = _midpoint(nn)
    p = _halo(a, nn, pbc, phases)
    for d in (1, 2, 3):
        n = a.shape[d]
        take = lambda o, m: p.narrow(d, nn + o, m)  # noqa: E731
        # even fine points are copies, odd ones midpoints; a zero-boundary axis
        # starts and ends with a midpoint
        lo, m = (0, n) if pbc else (-1, n + 1)
        odd = sum(w[j] * (take(lo - j, m) + take(lo + 1 + j, m)) for j in range(nn))
        even = take(0, n)
        if pbc:
            q = torch.stack((even, odd), d + 1).flatten(d, d + 1)
        else:
            q = torch.stack((odd.narrow(d, 0, n), even), d + 1).flatten(d, d + 1)
            q = torch.cat((q, odd.narrow(d, n, 1)), d)
        p = q
    return p


def _solve(gd, n, pbc, nn, relax, rho):
    """The multigrid solve: (phi, V-cycles)."""
    h0 = 0.2 / BOHR
    grids = [tuple(n)]
    while len(grids) < 5 and not any(x % 2 for x in grids[-1]) and \
            (pbc or all(x // 2 > 1 for x in grids[-1])):
        grids.append(tuple(x // 2 for x in grids[-1]))
    last = len(grids) - 1
    terms = [_laplace_terms({}, g, -0.25 / math.pi, nn if lv == 0 else 1, h0 * 2 ** lv)
             for lv, g in enumerate(grids)]
    pre = [2] + [4] * last
    post = [1] + [4] * last
    weight = [2.0 / 3.0] + [1.0] * last
    post[last] = 8

    def smooth(phi, src, lv, sweeps):
        if relax == 'J':
            c0 = terms[lv][0][1]
            for _ in range(sweeps):
                phi = phi + weight[lv] / c0 * (src - _stencil(phi, terms[lv], pbc))
            return phi
        colours = 4 if (nn if lv == 0 else 1) == 3 else 3 if (nn if lv == 0 else 1) == 2 else 2
        idx = sum(torch.meshgrid(*[torch.arange(x, device=phi.device) for x in phi.shape[1:]],
                                 indexing='ij')) % colours
        c0 = terms[lv][0][1]
        width = max(max(abs(x) for x in o) for o, _ in terms[lv])
        for _ in range(sweeps):
            p = _halo(phi, width, pbc)  # the halo is filled once per sweep
            inner = (slice(None),) + tuple(slice(width, width + x) for x in phi.shape[1:])
            for c in range(colours):
                s = torch.zeros_like(phi)
                for o, w in terms[lv][1:]:
                    s += w * p[(slice(None),) + tuple(
                        slice(width + int(x), width + int(x) + m) for x, m in zip(o, phi.shape[1:]))]
                p[inner] = torch.where(idx == c, (src - s) / c0, p[inner])
            phi = p[inner].clone()
        return phi

    def cycle(phi, src, lv):
        if lv < last:
            phi = smooth(phi, src, lv, pre[lv])
            r = _restrict(_stencil(phi, terms[lv], pbc) - src, 1, pbc)
            phi = phi - _interpolate(cycle(torch.zeros_like(r), r, lv + 1), 1, pbc)
        return smooth(phi, src, lv, post[lv])

    dv = h0 ** 3
    src = (rho - rho.sum() / math.prod(n if pbc else [x for x in rho.shape]))[None]
    phi = torch.zeros_like(src)
    for it in range(1, 1001):
        phi = cycle(phi, src, 0)
        r = _stencil(phi, terms[0], pbc) - src
        if float((r * r).sum()) * dv <= EPS:
            break
    if pbc:
        phi = phi - phi.mean()
    return phi[0], it


def _by_bands(f, x, chunk):
    return torch.cat([f(x[b:b + chunk]) for b in range(0, x.shape[0], chunk)])


def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def exact(case, seed):
    kind = case['kind']
    if kind == 'poisson':
        gd = _gd(case, 0.2 / BOHR)
        rho = _gaussians(gd, case['charges'], seed)
        phi, it = _solve(gd, _n(case), case['pbc'], case['nn'], case['relax'], rho)
        return {'phi': phi, 'niter': it}
    if kind == 'batch':
        phis, its = [], []
        for i, n in enumerate(_batch_sizes(case)):
            if i >= len(case['sizes'].split(',')):
                phis.append(None)  # one solve of each size
                its.append(None)
                continue
            gd = GridDescriptor((n,) * 3, (n * 0.2 / BOHR,) * 3, False)
            rho = _gaussians(gd, case['charges'], 1000 * seed + i)
            phi, it = _solve(gd, (n, n, n), False, case['nn'], case['relax'], rho)
            phis.append(phi)
            its.append(it)
        return {'phi': phis, 'niter': its}
    n, nn, pbc = _n(case), case['nn'], case['pbc']
    chunk = max(1, int(2e7 // math.prod(n)))
    if kind in ('laplace', 'gradient', 'hamiltonian', 'skew'):
        gd, ph = _gd(case), _phases(case)
        x = _bands(gd, case, seed)
        if kind == 'gradient':
            h = 0.18 / BOHR
            out = []
            for v in range(3):
                e = np.eye(3, dtype=int)[v]
                terms = []
                for m, w in enumerate(_first(nn), 1):
                    terms += [(tuple(m * e), w / h), (tuple(-m * e), -w / h)]
                out.append(_by_bands(lambda a: _stencil(_wide(a), terms, pbc, ph), x, chunk))
            return out
        terms = _laplace_terms(case, n, -0.5, nn)
        if kind == 'hamiltonian':
            real = torch.float32 if case['dtype'] in ('float32', 'complex64') else torch.float64
            vt = torch.randn(tuple(int(m) for m in gd.n_c), dtype=real, device='cuda',
                             generator=_gen(seed + 1)).double()
            f = lambda a: _stencil(_wide(a), terms, pbc, ph) + vt * _wide(a)  # noqa: E731
        else:
            f = lambda a: _stencil(_wide(a), terms, pbc, ph)  # noqa: E731
        return [_by_bands(f, x, chunk)]
    if kind == 'precondition':
        gd, ph = _gd(case), _phases(case)
        h = 0.18 / BOHR
        kin = [_laplace_terms(case, n, -0.5, nn if lv == 0 else 1, h * 2 ** lv) for lv in range(3)]
        step = 0.66666666 / kin[0][0][1]

        def f(R):
            apply = lambda lv, a: _stencil(a, kin[lv], pbc, ph)  # noqa: E731
            r1 = _restrict(-R, 1, pbc, ph)
            d1 = 4 * step * r1
            r2 = _restrict(apply(1, d1) - r1, 1, pbc, ph)
            d2 = 16 * step * r2
            d2 = d2 - 16 * step * (apply(2, d2) - r2)
            d1 = d1 - _interpolate(d2, 1, pbc, ph)
            d1 = d1 - 4 * step * (apply(1, d1) - r1)
            d0 = _interpolate(-d1, 1, pbc, ph)
            return step * (apply(0, d0) - R) - d0

        return _by_bands(lambda a: f(_wide(a)), _bands(gd, case, seed), chunk)
    coarse = _gd(case, 0.2 / BOHR)
    gd = coarse.refine() if kind == 'restrict' else coarse
    x = _bands(gd, case, seed)
    chunk = max(1, chunk // 8)
    if kind == 'restrict':
        return _by_bands(lambda a: _restrict(_wide(a), nn, pbc), x, chunk)
    if kind == 'interpolate':
        return _by_bands(lambda a: _interpolate(_wide(a), nn, pbc), x, chunk)
    y = _by_bands(lambda a: _interpolate(a, nn, pbc), x.abs_(), chunk)
    if not pbc:
        y *= _charge(case) / (y.sum() * coarse.refine().dv)
    return y
