"""Performance cases of the grid hot path.

What a real-space DFT program has this package do, through the package's
public entry points, on device-resident arrays:

  kinetic       T psi + v psi of a block of bands (nn=3 Laplacian, scale -1/2)
  gradient      an nn=3 gradient of a block of bands
  laplace_hex   the nn=3 Laplacian of a hexagonal cell (diagonal directions)
  interpolate   spin densities from the coarse to the fine grid (nn=3)
  restrict      effective potentials from the fine to the coarse grid (nn=3)
  precondition  the eigensolver's three-grid preconditioner on a band block
  overlap       the matrix sum(conj(a_x) b_y) dv of two band blocks
  poisson       multigrid Poisson solves to a relative residual of 1e-10

`listed` gives the measured cases, `draw` further ones of the same ranges;
`prepare`, `run`, `work`, `tolerance` and `exact` serve both.
"""
import math

import numpy as np
import torch

H = 0.38            # grid spacing, Bohr (0.2 Angstrom)
K_C = (0.2, -0.3, 0.45)   # k-point of the Bloch cases, reciprocal units
REL = 1e-10         # relative residual of the Poisson solves
LAPL3 = {0: -49 / 18, 1: 3 / 2, 2: -3 / 20, 3: 1 / 90}
LAPL1 = {0: -2.0, 1: 1.0}
GRAD3 = {1: 3 / 4, 2: -3 / 20, 3: 1 / 60}
ES = {'float64': 8, 'complex128': 16, 'float32': 4, 'complex64': 8}


def _case(name, kind, dtype, pbc, n, count, **more):
    c = {'kind': kind, 'dtype': dtype, 'pbc': pbc, 'N0': n[0], 'N1': n[1],
         'N2': n[2], 'count': count}
    if name:
        c['name'] = name
    c.update(more)
    return c


def listed():
    return [
        # one small molecule's few bands: latency of a single call
        _case('kinetic_small_f64', 'kinetic', 'float64', False,
              (32, 32, 32), 4),
        # a molecule in a box: real bands, zero boundaries, hence odd rows
        _case('kinetic_molecule_f64', 'kinetic', 'float64', False,
              (96, 96, 96), 48),
        # a bulk k-point: complex bands with Bloch phases
        _case('kinetic_bloch_c128', 'kinetic', 'complex128', True,
              (96, 96, 96), 48),
        # the same in single precision, on a non-cubic cell
        _case('kinetic_bloch_c64', 'kinetic', 'complex64', True,
              (84, 90, 108), 64),
        # momentum matrix elements: a gradient of the bands of a slab cell
        _case('gradient_bloch_c128', 'gradient', 'complex128', True,
              (80, 72, 88), 32, axis=1),
        # a layered material in its hexagonal cell
        _case('laplace_hex_c128', 'laplace_hex', 'complex128', True,
              (60, 60, 84), 24),
        # two spin densities of a molecule to the fine grid
        _case('interpolate_density_f64', 'interpolate', 'float64', False,
              (96, 96, 96), 2),
        # two spin potentials of a bulk cell to the coarse grid
        _case('restrict_potential_f64', 'restrict', 'float64', True,
              (96, 96, 96), 2),
        # the residuals of one block of an eigensolver iteration
        _case('precondition_bloch_c128', 'precondition', 'complex128', True,
              (72, 72, 72), 16),
        # the subspace matrix of one k-point
        _case('overlap_c128', 'overlap', 'complex128', True,
              (56, 56, 56), 48),
        # the Hartree potential of a bulk cell, once per SCF step
        _case('poisson_bulk_f64', 'poisson', 'float64', True,
              (80, 80, 80), 1, precision='fp64'),
        # many independent molecules' Hartree potentials at once
        _case('poisson_batch_fp32', 'poisson', 'float64', False,
              (128, 128, 128), 16, precision='fp32'),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['kinetic', 'kinetic', 'gradient', 'laplace_hex',
                       'interpolate', 'restrict', 'precondition', 'overlap',
                       'poisson'])
    pbc = rng.random() < 0.6
    if kind == 'poisson':
        n = [8 * rng.randint(4, 14) for _ in range(3)]
        prec = rng.choice(['fp64', 'fp32'])
        if prec == 'fp32':
            pbc = False
        points = n[0] * n[1] * n[2]
        most = max(1, min(12, (4 if prec == 'fp64' else 12) * 96 ** 3 //
                          points))
        return _case('', kind, 'float64', pbc, n, _logint(rng, 1, most),
                     precision=prec)
    if kind == 'interpolate' or kind == 'restrict':
        # (coarse grid; real densities and potentials)
        n = [rng.randint(12, 90) for _ in range(3)]
        return _case('', kind, 'float64', pbc, n, rng.randint(1, 2))
    if kind == 'precondition':
        n = [4 * rng.randint(6, 20) for _ in range(3)]
    elif kind == 'laplace_hex':
        a = rng.randint(16, 64)
        n = [a, a, rng.randint(16, 90)]
        pbc = True
    elif kind == 'overlap':
        n = [rng.randint(12, 56) for _ in range(3)]
    else:
        n = [rng.randint(14, 112) for _ in range(3)]
    # complex bands carry Bloch phases: periodic cells only
    dtype = rng.choice(['complex128', 'complex128', 'complex64', 'float64']) \
        if pbc else rng.choice(['float64', 'float64', 'float32'])
    if kind == 'overlap' and dtype in ('complex64', 'float32'):
        dtype = 'complex128' if pbc else 'float64'
    points = n[0] * n[1] * n[2]
    most = 40 * 96 ** 3 * 16 // (points * ES[dtype])
    most = max(2, min(48 if kind == 'overlap' else 64, most))
    if kind == 'laplace_hex' or kind == 'precondition':
        most = max(2, min(most, 24 * 72 ** 3 // points))
    more = {'axis': rng.randint(0, 2)} if kind == 'gradient' else {}
    return _case('', kind, dtype, pbc, n, _logint(rng, 1, most), **more)


# ------------------------------------------------------------------ inputs
def _N(case):
    return (case['N0'], case['N1'], case['N2'])


def _cell(case):
    n = _N(case)
    if case['kind'] == 'laplace_hex':
        a, c = H * n[0], H * n[2]
        return [(a, 0.0, 0.0), (-0.5 * a, 0.5 * math.sqrt(3.0) * a, 0.0),
                (0.0, 0.0, c)]
    return tuple(H * m for m in n)


def _extent(case, fine=False):
    m = 2 if fine else 1
    return tuple(m * n - (0 if case['pbc'] else 1) for n in _N(case))


def _phases(case):
    if not case['dtype'].startswith('complex'):
        return None
    # psi(r + R) = exp(2 pi i k.R) psi(r): [c, 0] above, [c, 1] below the cell
    k = np.array(K_C)[:, np.newaxis] * np.array([1.0, -1.0])
    return np.exp(2j * np.pi * k)


def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _randn(shape, dtype, gen):
    return torch.randn(shape, dtype=getattr(torch, dtype), device='cuda',
                       generator=gen)


def _density(case, seed):
    """Neutral sums of 8 Gaussians of charge +-1 per grid, float64."""
    rng = np.random.default_rng([int(seed), 7])
    ext = _extent(case)
    beg = 0 if case['pbc'] else 1
    box = [H * n for n in _N(case)]
    x = [(torch.arange(n, dtype=torch.float64, device='cuda') + beg) * H
         for n in ext]
    rho = torch.zeros((case['count'],) + ext, dtype=torch.float64,
                      device='cuda')
    for b in range(case['count']):
        for i in range(8):
            s = rng.uniform(0.95, 2.8)
            g = []
            for c in range(3):
                d = x[c] - rng.uniform(0.25, 0.75) * box[c]
                if case['pbc']:
                    d = d - box[c] * torch.round(d / box[c])
                g.append(torch.exp(-d ** 2 / (2 * s * s)))
            q = (1.0 if i % 2 == 0 else -1.0) * (2 * math.pi * s * s) ** -1.5
            rho[b] += q * (g[0][:, None, None] * g[1][None, :, None] *
                           g[2][None, None, :])
        rho[b] -= rho[b].mean()
    return rho


def _inputs(case, seed):
    kind = case['kind']
    if kind == 'poisson':
        return {'rho': _density(case, seed)}
    gen = _generator(seed)
    shape = (case['count'],) + _extent(case, kind == 'restrict')
    s = {'a': _randn(shape, case['dtype'], gen)}
    if kind == 'kinetic':
        real = 'float64' if case['dtype'] in ('float64', 'complex128') \
            else 'float32'
        s['v'] = _randn(shape[1:], real, gen)
    if kind == 'overlap':
        # H psi: close to a multiple of psi, as in an eigensolver
        s['b'] = _randn(shape, case['dtype'], gen).mul_(0.1).add_(s['a'])
    return s


# ------------------------------------------------------------------ the path
def prepare(case, seed):
    from gpawdft_b200.fd_operators import Gradient, Laplace
    from gpawdft_b200.grid_descriptor import GridDescriptor
    from gpawdft_b200.poisson import PoissonSolver
    from gpawdft_b200.preconditioner import Preconditioner
    from gpawdft_b200.transformers import Transformer
    kind, dtype = case['kind'], np.dtype(case['dtype'])
    gd = GridDescriptor(_N(case), _cell(case), case['pbc'])
    s = _inputs(case, seed)
    s['kind'] = kind
    s['phases'] = _phases(case)
    if kind == 'kinetic':
        s['op'] = Laplace(gd, -0.5, 3, dtype)
        s['out'] = torch.empty_like(s['a'])
    elif kind == 'gradient':
        s['op'] = Gradient(gd, case['axis'], 1.0, 3, dtype)
        s['out'] = torch.empty_like(s['a'])
    elif kind == 'laplace_hex':
        s['op'] = Laplace(gd, -0.5, 3, dtype)
        s['out'] = torch.empty_like(s['a'])
    elif kind == 'interpolate' or kind == 'restrict':
        fine = gd.refine()
        s['op'] = Transformer(gd, fine, 3, dtype) if kind == 'interpolate' \
            else Transformer(fine, gd, 3, dtype)
        s['out'] = torch.empty((case['count'],) +
                               _extent(case, kind == 'interpolate'),
                               dtype=s['a'].dtype, device='cuda')
    elif kind == 'precondition':
        s['op'] = Preconditioner(gd, Laplace(gd, -0.5, 3, dtype), dtype,
                                 case['count'])
    elif kind == 'overlap':
        s['gd'] = gd
    else:
        ps = PoissonSolver(nn=3, relax='J', precision=case['precision'],
                           batch=case['count'])
        ps.set_grid_descriptor(gd)
        ps.initialize()
        s['op'] = ps
        s['eps'] = (REL ** 2 * gd.dv *
                    (s['rho'] ** 2).sum(dim=(1, 2, 3))).cpu().numpy()
        s['phi'] = torch.empty_like(s['rho'])
    return s


def run(s):
    kind = s['kind']
    if kind == 'kinetic':
        s['op'].apply_potential(s['a'], s['out'], s['v'], s['phases'])
        return s['out']
    if kind == 'gradient' or kind == 'laplace_hex':
        s['op'].apply(s['a'], s['out'], s['phases'])
        return s['out']
    if kind == 'interpolate' or kind == 'restrict':
        return s['op'].apply(s['a'], s['out'], s['phases'])
    if kind == 'precondition':
        return s['op'](s['a'], s['phases'])
    if kind == 'overlap':
        return s['gd'].integrate(s['a'], s['b'])
    # poisson: from a zero potential, each grid to its own tolerance
    s['phi'].zero_()
    if s['phi'].shape[0] == 1:
        s['op'].solve(s['phi'][0], s['rho'][0], eps=float(s['eps'][0]))
    else:
        s['op'].solve_batch(s['phi'], s['rho'], eps=s['eps'])
    return s['phi']


def work(case):
    kind, es = case['kind'], ES[case['dtype']]
    comp = 2 if case['dtype'].startswith('complex') else 1
    coarse = case['count'] * math.prod(_extent(case))
    fine = case['count'] * math.prod(_extent(case, True))
    if kind == 'kinetic':
        v = math.prod(_extent(case)) * es // comp
        return {'bytes': 2 * es * coarse + v, 'flops': 40 * comp * coarse}
    if kind == 'gradient':
        return {'bytes': 2 * es * coarse, 'flops': 12 * comp * coarse}
    if kind == 'laplace_hex':
        # 1 + 6 x 4 points: three in-plane directions and the axis
        return {'bytes': 2 * es * coarse, 'flops': 50 * comp * coarse}
    if kind == 'interpolate':
        # three 1D passes of 6 taps on every second point of an axis
        return {'bytes': es * (coarse + fine), 'flops': 8 * comp * 2 * fine}
    if kind == 'restrict':
        return {'bytes': es * (coarse + fine), 'flops': 10 * comp * fine}
    if kind == 'precondition':
        # the fine-grid kinetic apply, and the coarse grids (1/8 each) and
        # transfers at about half as much again
        return {'bytes': 2 * es * coarse, 'flops': 60 * comp * coarse}
    if kind == 'overlap':
        return {'bytes': 2 * es * coarse,
                'flops': (8 if comp == 2 else 2) * case['count'] * coarse}
    # poisson: rho read and phi written once; ten digits at about one per
    # V-cycle of two sweeps and a residual (19 points) and their coarse levels
    return {'bytes': 2 * 8 * coarse, 'flops': 10 * 3 * 38 * 8 / 7 * coarse}


def tolerance(case):
    kind = case['kind']
    if kind == 'poisson':
        # two solves that both stop at this residual: the potential is off
        # the exact one by 4e-11 (fp32) and 5e-13 to 3e-12 (fp64)
        return {'rel': 1.5e-10 if case['precision'] == 'fp32' else 2e-11}
    if case['dtype'] in ('float32', 'complex64'):
        return {'rel': 4e-7}      # 1e-7 off the exact result
    if kind == 'overlap':
        return {'rel': 3e-15}     # 6e-16
    return {'rel': 2e-15}         # 1e-16 to 6e-16


# ------------------------------------------------------------------ 64 bits
def _shift(a, axis, s, pbc, phases):
    """a[i + s] along a grid axis (0 - 2), with its boundary."""
    d = axis - 3
    r = torch.roll(a, -s, d)
    n = a.shape[d]
    m = min(abs(s), n)
    edge = r.narrow(d, n - m, m) if s > 0 else r.narrow(d, 0, m)
    if not pbc:
        edge.zero_()
    elif phases is not None:
        edge.mul_(complex(phases[axis][0 if s > 0 else 1]))
    return r


def _star(a, table, h, scale, pbc, phases):
    """scale * sum over the axes of table[|s|] a[i + s] / h^2."""
    out = a * (3 * scale * table[0] / h ** 2)
    for axis in range(3):
        for s, w in table.items():
            if s:
                for t in (s, -s):
                    out.add_(_shift(a, axis, t, pbc, phases),
                             alpha=scale * w / h ** 2)
    return out


def _take(a, axis, idx, N, pbc, phases):
    """Values at global indices idx of a grid of N points per period (stored
    from 0 when periodic, from 1 with zeros outside otherwise)."""
    d = axis - 3
    if pbc:
        r = a.index_select(d, idx % N)
        if phases is None:
            return r
        f = torch.ones(len(idx), dtype=a.dtype, device=a.device)
        f[idx >= N] = complex(phases[axis][0])
        f[idx < 0] = complex(phases[axis][1])
    else:
        ok = (idx >= 1) & (idx <= N - 1)
        r = a.index_select(d, (idx - 1).clamp(0, N - 2))
        f = ok.to(a.dtype)
    shape = [1, 1, 1]
    shape[axis] = len(idx)
    return r * f.reshape(shape)


W_MID = {1: (0.5,), 3: (0.5859375, -0.09765625, 0.01171875)}


def _interp(a, n, nn, pbc, phases):
    for axis in range(3):
        N = n[axis]
        g = torch.arange(0 if pbc else 1, 2 * N, device=a.device)
        i = g // 2
        even = _take(a, axis, i, N, pbc, phases)
        mid = 0
        for j, w in enumerate(W_MID[nn]):
            mid = mid + w * (_take(a, axis, i - j, N, pbc, phases) +
                             _take(a, axis, i + 1 + j, N, pbc, phases))
        shape = [1, 1, 1]
        shape[axis] = len(g)
        a = torch.where((g % 2 == 0).reshape(shape), even, mid)
    return a


def _restr(a, n, nn, pbc, phases):
    """From 2 n to n points per period."""
    for axis in range(3):
        N = n[axis]
        i = 2 * torch.arange(0 if pbc else 1, N, device=a.device)
        out = _take(a, axis, i, 2 * N, pbc, phases)
        for j, w in enumerate(W_MID[nn]):
            out = out + w * (
                _take(a, axis, i - 2 * j - 1, 2 * N, pbc, phases) +
                _take(a, axis, i + 2 * j + 1, 2 * N, pbc, phases))
        a = 0.5 * out
    return a


def _precondition(r, n, pbc, ph):
    def kin(x, level):
        return _star(x, LAPL1 if level else LAPL3, H * 2 ** level, -0.5, pbc,
                     ph)
    n1 = [m // 2 for m in n]
    n2 = [m // 4 for m in n]
    step = 0.66666666 / (-0.5 * 3 * LAPL3[0] / H ** 2)
    r1 = _restr(-r, n1, 1, pbc, ph)
    d1 = 4 * step * r1
    r2 = _restr(kin(d1, 1) - r1, n2, 1, pbc, ph)
    d2 = 16 * step * r2
    d2 = d2 - 16 * step * (kin(d2, 2) - r2)
    d1 = d1 - _interp(d2, n2, 1, pbc, ph)
    d1 = d1 - 4 * step * (kin(d1, 1) - r1)
    d0 = _interp(-d1, n1, 1, pbc, ph)
    return -(d0 - step * (kin(d0, 0) - r))


def _poisson(rho, pbc):
    """Conjugate gradients on -laplace / (4 pi) with the nn=3 stencil."""
    dims = (1, 2, 3)
    rho = rho - rho.mean(dim=dims, keepdim=True)
    phi = torch.zeros_like(rho)
    r, p = rho.clone(), rho.clone()
    rr = (r * r).sum(dim=dims, keepdim=True)
    stop = rr * 1e-28
    for _ in range(4000):
        q = _star(p, LAPL3, H, -0.25 / math.pi, pbc, None)
        alpha = torch.where(rr > stop, rr / (p * q).sum(dim=dims,
                                                        keepdim=True), 0.0)
        phi += alpha * p
        r -= alpha * q
        new = (r * r).sum(dim=dims, keepdim=True)
        if bool((new <= stop).all()):
            break
        p = r + (new / rr) * p
        rr = new
    if pbc:
        phi -= phi.mean(dim=dims, keepdim=True)
    return phi


def exact(case, seed):
    kind, pbc, n = case['kind'], case['pbc'], _N(case)
    s = _inputs(case, seed)
    ph = _phases(case)
    if kind == 'poisson':
        return _poisson(s['rho'], pbc)
    wide = torch.complex128 if ph is not None else torch.float64
    a = s['a'].to(wide)
    if kind == 'kinetic':
        return _star(a, LAPL3, H, -0.5, pbc, ph) + s['v'].double() * a
    if kind == 'gradient':
        out = torch.zeros_like(a)
        for m, w in GRAD3.items():
            out.add_(_shift(a, case['axis'], m, pbc, ph), alpha=w / H)
            out.sub_(_shift(a, case['axis'], -m, pbc, ph), alpha=w / H)
        return out
    if kind == 'laplace_hex':
        # 2 / 3 of the second differences along a, b and a + b, and that
        # along c
        out = a * (-0.5 * (3 * 2 / 3 + 1) * LAPL3[0] / H ** 2)
        for m in (1, 2, 3):
            for t in (m, -m):
                w = -0.5 * LAPL3[m] / H ** 2
                x = _shift(a, 0, t, pbc, ph)
                out.add_(x, alpha=2 / 3 * w)
                out.add_(_shift(x, 1, t, pbc, ph), alpha=2 / 3 * w)
                out.add_(_shift(a, 1, t, pbc, ph), alpha=2 / 3 * w)
                out.add_(_shift(a, 2, t, pbc, ph), alpha=w)
        return out
    if kind == 'interpolate':
        return _interp(a, n, 3, pbc, ph)
    if kind == 'restrict':
        return _restr(a, n, 3, pbc, ph)
    if kind == 'precondition':
        return _precondition(a, n, pbc, ph)
    # overlap
    dv = H ** 3
    x, y = a.flatten(1), s['b'].to(wide).flatten(1)
    return (torch.conj(x) @ y.T * dv).cpu().numpy()
