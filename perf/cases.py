"""Timed workloads of the finite-difference path, each one pass through the
public entry points, with the inputs a calculation has at that point.

Kinds (the "kind" entry of a case):
  kinetic   Laplace(gd, -1/2, 3): apply, or apply_potential (T + v) psi
  vcycle    the multigrid preconditioner on a block of residuals
  transfer  density to the fine grid and potential back to the coarse one
  residual  projections of the wave functions, then H psi - eps psi + sum p dH P
  xc        XC('PBE').calculate on the fine grid
  rmmdiis   one RMM-DIIS pass over every band, orthonormalisation, density
  fold      the learned preconditioner's inference form
  train     one training step of it: forward, loss, gradients
Grids are given as N (grid points per axis, GridDescriptor's N_c); a
zero-boundary grid has N - 1 points per axis.
"""
from math import gamma, pi, sqrt
from types import SimpleNamespace

import numpy as np
import torch
import torch.nn.functional as F

BOHR = 0.52917721
H = 0.2 / BOHR                # grid spacing of every case, 0.2 Angstrom
DTYPES = {'f64': torch.float64, 'f32': torch.float32,
          'c128': torch.complex128, 'c64': torch.complex64}
W2 = {1: [-2.0, 1.0], 3: [-49 / 18, 3 / 2, -3 / 20, 1 / 90]}   # d2/dx2, order 2 and 6
MID = {1: [0.5], 3: [75 / 128, -25 / 256, 3 / 256]}            # midpoint interpolation


def listed():
    return [
        # the H2 molecule in a box: four bands, a zero-boundary 31^3 grid --
        # the smallest calls of a calculation, latency and launches
        {'name': 'h2_kinetic', 'kind': 'kinetic', 'n0': 32, 'n1': 32, 'n2': 32, 'pbc': 0,
         'bands': 4, 'nk': 1, 'dtype': 'f64', 'potential': True},
        # the batched order-6 Laplacian of the benchmark
        {'name': 'laplace_256x96', 'kind': 'kinetic', 'n0': 96, 'n1': 96, 'n2': 96, 'pbc': 1,
         'bands': 256, 'nk': 1, 'dtype': 'f64', 'potential': False},
        # Bloch states: a batch of four k-points of an 8-atom cell
        {'name': 'kpoint_kinetic', 'kind': 'kinetic', 'n0': 28, 'n1': 28, 'n2': 28, 'pbc': 1,
         'bands': 24, 'nk': 4, 'dtype': 'c128', 'potential': True},
        # the preconditioner in the FP32 form on Si64 (56^3, 160 bands)
        {'name': 'si64_vcycle_f32', 'kind': 'vcycle', 'n0': 56, 'n1': 56, 'n2': 56, 'pbc': 1,
         'bands': 160, 'nk': 1, 'dtype': 'f32'},
        # the same in FP64 on (H2O)32 in a 15 A box: zero boundaries, the odd
        # 75^3 grid of a molecule
        {'name': 'water_vcycle_f64', 'kind': 'vcycle', 'n0': 76, 'n1': 76, 'n2': 76, 'pbc': 0,
         'bands': 160, 'nk': 1, 'dtype': 'f64'},
        # density and potential between the coarse and the fine grid, once per
        # SCF iteration: Si64 (56^3 and 112^3)
        {'name': 'si64_transfer', 'kind': 'transfer', 'n0': 56, 'n1': 56, 'n2': 56, 'pbc': 1,
         'grids': 1},
        # projections and residuals, FP32 form on Si64 with its HGH projectors
        {'name': 'si64_residual_f32', 'kind': 'residual', 'n0': 56, 'n1': 56, 'n2': 56, 'pbc': 1,
         'bands': 160, 'dtype': 'f32', 'atoms': 64, 'functions': 'hgh'},
        # the same in FP64, zero boundaries, s + p + d functions per atom
        {'name': 'cluster_residual_f64', 'kind': 'residual', 'n0': 72, 'n1': 72, 'n2': 72,
         'pbc': 0, 'bands': 96, 'dtype': 'f64', 'atoms': 24, 'functions': 'spd'},
        # PBE on the fine grid of (H2O)32
        {'name': 'water_pbe', 'kind': 'xc', 'n0': 152, 'n1': 152, 'n2': 152, 'pbc': 0,
         'spins': 1},
        # the whole eigensolver step, FP32 form on Si64
        {'name': 'si64_rmmdiis_f32', 'kind': 'rmmdiis', 'n0': 56, 'n1': 56, 'n2': 56, 'pbc': 1,
         'bands': 160, 'dtype': 'f32', 'atoms': 64},
        # the learned preconditioner: inference on Si64 and a training step
        {'name': 'si64_learned', 'kind': 'fold', 'n0': 56, 'n1': 56, 'n2': 56, 'bands': 160},
        {'name': 'si64_learned_train', 'kind': 'train', 'n0': 56, 'n1': 56, 'n2': 56, 'pbc': 1,
         'bands': 16},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo)**rng.random()))


def _sizes(rng, lo, hi, step=4):
    """Three grid sizes (multiples of `step`), the axes usually different."""
    n = _log(rng, lo, hi)
    return {f'n{c}': max(lo, step * round(n * rng.uniform(0.85, 1.15) / step))
            for c in range(3)}


def _bands(rng, grid, lo, hi, points):
    """A band count between lo and hi, at most `points` grid points in all."""
    n = grid['n0'] * grid['n1'] * grid['n2']
    return max(1, min(_log(rng, lo, hi), int(points / n)))


def draw(rng):
    kind = rng.choice(['kinetic', 'kinetic', 'vcycle', 'vcycle', 'transfer', 'residual', 'xc',
                       'rmmdiis', 'fold', 'train'])
    pbc = rng.randrange(2)
    if kind == 'kinetic':
        g = _sizes(rng, 20, 104, rng.choice([1, 2, 4]))
        dtype = rng.choice(['f64', 'f32', 'c128', 'c64'])
        nk = rng.choice([1, 2, 4]) if dtype[0] == 'c' else 1
        if dtype[0] == 'c':
            pbc = 1
        b = _bands(rng, g, 1, 200, 8e7) // nk
        return {'kind': kind, **g, 'pbc': pbc, 'bands': max(1, b), 'nk': nk, 'dtype': dtype,
                'potential': rng.random() < 0.7}
    if kind == 'vcycle':
        g = _sizes(rng, 24, 96)
        dtype = rng.choice(['f64', 'f32', 'f64', 'f32', 'c128'])
        nk = rng.choice([1, 4]) if dtype[0] == 'c' else 1
        if dtype[0] == 'c':
            pbc = 1
        b = _bands(rng, g, 1, 200, 4e7) // nk
        return {'kind': kind, **g, 'pbc': pbc, 'bands': max(1, b), 'nk': nk, 'dtype': dtype}
    if kind == 'transfer':
        return {'kind': kind, **_sizes(rng, 20, 96), 'pbc': pbc, 'grids': rng.choice([1, 1, 2])}
    if kind == 'residual':
        g = _sizes(rng, 36, 80)
        return {'kind': kind, **g, 'pbc': pbc, 'bands': _bands(rng, g, 1, 200, 3e7),
                'dtype': rng.choice(['f64', 'f32']), 'atoms': _log(rng, 2, 32),
                'functions': rng.choice(['hgh', 'spd'])}
    if kind == 'xc':
        return {'kind': kind, **_sizes(rng, 40, 160, 2), 'pbc': pbc, 'spins': rng.choice([1, 1, 2])}
    if kind == 'rmmdiis':
        g = _sizes(rng, 36, 64)
        return {'kind': kind, **g, 'pbc': pbc, 'bands': _bands(rng, g, 8, 160, 2e7),
                'dtype': rng.choice(['f64', 'f32']), 'atoms': _log(rng, 2, 24)}
    if kind == 'fold':
        g = _sizes(rng, 24, 72)
        return {'kind': kind, **g, 'bands': _bands(rng, g, 1, 200, 3e7)}
    g = _sizes(rng, 20, 56)
    return {'kind': 'train', **g, 'pbc': pbc, 'bands': rng.choice([4, 8, 16])}


# ---------------------------------------------------------------- inputs

def _n(case):
    return [case['n0'], case['n1'], case['n2']]


def _pbc(case):
    return bool(case.get('pbc', 1))


def _points(case):
    return [n - (0 if _pbc(case) else 1) for n in _n(case)]


def _rows(case):
    return case.get('bands', 1) * case.get('nk', 1)


def _dtype(case):
    return DTYPES[case.get('dtype', 'f64')]


def _gd(case, device='cuda'):
    from gpaw_b200.grid_descriptor import GridDescriptor
    return GridDescriptor(_n(case), np.array(_n(case)) * H, _pbc(case), device=device)


def _randn(shape, seed, dtype=torch.float64, part=0):
    g = torch.Generator(device='cuda').manual_seed(1000003 * part + seed)
    return torch.randn(shape, generator=g, device='cuda', dtype=dtype)


def _phases(case, seed):
    """(nk, 3, 2) Bloch phases exp(+-2 pi i k_c) of nk k-points, or one
    (3, 2) set, or None for real data."""
    if not _dtype(case).is_complex:
        return None
    k = np.random.default_rng(seed).uniform(-0.5, 0.5, (case['nk'], 3))
    ph = np.exp(2j * np.pi * k[:, :, None] * np.array([1.0, -1.0]))
    return ph if case['nk'] > 1 else ph[0]


def _waves(case, seed, part=0):
    """Smooth band-like fields: a few low plane (or sine) waves per band plus
    noise at a tenth of their size."""
    nb, n, N = _rows(case), _points(case), _n(case)
    rng = np.random.default_rng(seed + 7919 * part)
    psi = 0.1 * _randn((nb, *n), seed, torch.float32, part).to(torch.float64)
    for _ in range(2):
        f = []
        for c in range(3):
            if _pbc(case):
                x = 2 * pi * np.arange(n[c]) / N[c]
                m = rng.integers(0, 5, nb)[:, None]
                w = np.cos(m * x + rng.uniform(0, 2 * pi, (nb, 1)))
            else:
                w = np.sin(rng.integers(1, 7, nb)[:, None] * pi * np.arange(1, n[c] + 1) / N[c])
            f.append(torch.from_numpy(w).cuda())
        psi += f[0][:, :, None, None] * f[1][:, None, :, None] * f[2][:, None, None, :]
    return psi


def _atoms(case, seed):
    """Scaled positions: a jittered lattice that fills the cell (clear of the
    walls of a zero-boundary box)."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(case['atoms']**(1 / 3)))
    p = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing='ij'), -1).reshape(-1, 3)
    p = (rng.permutation(p)[:case['atoms']] + 0.5 + rng.uniform(-0.1, 0.1, (case['atoms'], 3))) / m
    return p if _pbc(case) else 0.2 + 0.6 * p


def _radials(functions):
    """[(l, cutoff, table)]: the HGH projectors of Si (two s, two p), or one
    Gaussian each of s, p and d with a 2.5 Angstrom cutoff."""
    out = []
    if functions == 'hgh':
        for l, rl in ((0, 0.422738), (1, 0.484278)):
            rc = rl * sqrt(90.0)
            r = np.linspace(0, rc, 401)
            for i in (1, 2):
                a = l + (4 * i - 1) / 2.0
                f = sqrt(2.0) / (rl**a * sqrt(gamma(a))) * r**(2 * (i - 1)) * np.exp(-0.5 * (r / rl)**2)
                f[-1] = 0.0
                out.append((l, rc, f))
    else:
        rc = 2.5 / BOHR
        r = np.linspace(0, rc, 101)
        for l in (0, 1, 2):
            f = np.exp(-(r / (0.8 / BOHR))**2)
            f[-1] = 0.0
            out.append((l, rc, f))
    return out


def _dh(functions):
    """The atomic Hamiltonian in the functions' order (HGH Si values, or a
    diagonal)."""
    if functions == 'hgh':
        s = np.array([[5.906928, -0.5 * sqrt(3 / 5) * 3.258196],
                      [-0.5 * sqrt(3 / 5) * 3.258196, 3.258196]])
        d = np.zeros((8, 8))
        d[:2, :2] = s
        d[2:5, 2:5] = 2.727013 * np.eye(3)
        return d
    return np.diag(np.linspace(0.5, -0.5, 9))


def _dh_matrix(case, functions):
    d = torch.from_numpy(_dh(functions)).cuda()
    return torch.block_diag(*[d] * case['atoms'])


def _splines(functions):
    from gpaw_b200.spline import Spline
    return [Spline.from_data(l, rc, f) for l, rc, f in _radials(functions)]


def _density(case, seed):
    """Electron density of Gaussian atoms (width 1 bohr, six electrons each,
    about one atom per 230 bohr^3 of a molecular box), decaying to nothing
    at the walls: (spins, n0, n1, n2)."""
    rng = np.random.default_rng(seed)
    n, N = _points(case), _n(case)
    h = H / 2 if case['kind'] == 'xc' else H      # XC and transfers run on the fine grid's spacing
    L = np.array(N) * h
    natoms = max(2, int(np.prod(L) / 230.0))
    pos = rng.uniform(0.15, 0.85, (natoms, 3)) * L
    out = []
    for s in range(case.get('spins', 1)):
        f = []
        for c in range(3):
            x = (np.arange(n[c]) + (0 if _pbc(case) else 1)) * h
            d = x[None] - pos[:, c:c + 1]
            if _pbc(case):
                d -= L[c] * np.round(d / L[c])
            f.append(torch.from_numpy(np.exp(-0.5 * d * d)).cuda())
        q = torch.from_numpy(rng.uniform(2.0, 4.0, natoms) / (2 * pi)**1.5).cuda()
        out.append(torch.einsum('a,ax,ay,az->xyz', q, *f))
    return torch.stack(out)


def _params(seed):
    """The network's weights after some training: the V-cycle-like magnitudes
    of its layers, seeded."""
    rng = np.random.default_rng(seed)
    out = {}
    for k, (co, ci) in {'w0': (1, 1), 'wa': (16, 1), 'wb': (16, 16), 'wc': (1, 16),
                        'wp': (1, 1)}.items():
        w = rng.standard_normal((co, ci, 27)) / sqrt(27 * ci)
        if k in ('w0', 'wp'):
            w[0, 0, 13] += 1.0
        out[k] = torch.from_numpy(w).float().cuda()
    return out


# ---------------------------------------------------------------- the passes

def prepare(case, seed):
    kind = case['kind']
    gd = _gd(case)
    s = SimpleNamespace(kind=kind, gd=gd)
    dt = _dtype(case)
    cplx = complex if dt.is_complex else float
    shape = (_rows(case), *_points(case))
    if kind == 'kinetic':
        from gpaw_b200.fd_operators import Laplace
        s.op = Laplace(gd, -0.5, 3, cplx)
        s.x = _randn(shape, seed, dt)
        s.y = torch.empty_like(s.x)
        s.phases = _phases(case, seed)
        real = torch.float32 if dt in (torch.float32, torch.complex64) else torch.float64
        s.v = _randn(shape[1:], seed, torch.float64, 1).to(real) if case['potential'] else None
    elif kind == 'vcycle':
        from gpaw_b200.fd_operators import Laplace
        from gpaw_b200.preconditioner import Preconditioner
        s.pc = Preconditioner(gd, Laplace(gd, -0.5, 3, cplx), cplx, block=10)
        s.R = _randn(shape, seed, dt)
        ph = _phases(case, seed)
        s.kpt = None if ph is None else SimpleNamespace(phase_cd=ph)
    elif kind == 'transfer':
        from gpaw_b200.transformers import Transformer
        fine = gd.refine()
        s.up, s.down = Transformer(gd, fine, 3), Transformer(fine, gd, 3)
        s.n = torch.cat([_density(case, seed + i) for i in range(case['grids'])])
        s.v = _randn((case['grids'], *fine.n_c.tolist()), seed)
    elif kind == 'residual':
        from gpaw_b200.lfc import LFC
        s.pt = LFC(gd, [_splines(case['functions'])] * case['atoms'], cut=True)
        s.pt.set_positions(_atoms(case, seed))
        s.dH = _dh_matrix(case, case['functions']).to(dt)
        s.psi, s.Hpsi = _waves(case, seed).to(dt), _waves(case, seed, 1).to(dt)
        e = torch.linspace(-0.4, 0.3, shape[0], dtype=torch.float64, device='cuda')
        s.coef = torch.stack([torch.ones_like(e), -e], 1)
    elif kind == 'xc':
        from gpaw_b200.grid_descriptor import GridDescriptor
        from gpaw_b200.xc import XC
        s.gd = GridDescriptor(_n(case), np.array(_n(case)) * H / 2, _pbc(case))
        s.xc = XC('PBE')
        s.xc.set_grid_descriptor(s.gd)
        s.n = _density(case, seed)
    elif kind == 'rmmdiis':
        _prepare_rmmdiis(s, case, seed, dt)
    else:
        from gpaw_b200.learned import ConvNet, FoldedNet
        params = _params(seed)
        s.net = ConvNet(gd, params=params)
        s.R = _randn(shape, seed, torch.float32)
        if kind == 'fold':
            s.folded = FoldedNet(s.net, scale=0.05)
        else:
            s.T = _randn(shape, seed, torch.float32, 1)
    return s


def _prepare_rmmdiis(s, case, seed, dt):
    from gpaw_b200.eigensolvers import RMMDIIS
    from gpaw_b200.preconditioner import Preconditioner
    from gpaw_b200.wavefunctions import FDWaveFunctions
    nb = case['bands']
    sp = _splines('hgh')
    setup = SimpleNamespace(pt_j=sp, ni=8, dH_ii=_dh('hgh'))
    s.wfs = FDWaveFunctions(s.gd, nb, [setup] * case['atoms'], _atoms(case, seed), dt, 3)
    s.es = RMMDIIS()
    s.es.initialize(s.wfs, Preconditioner(s.gd, s.wfs.kin, float, block=10))
    psi, v, eps, V, P, f, w = _rmmdiis_inputs(case, seed, dt)
    s.psi, s.eps, s.V, s.f, s.w = psi, eps, V, f, w
    s.P = P.to(dt)
    s.ham = SimpleNamespace(vt_G=v, vt_G32=v.to(torch.float32), dH_MM=_dh_matrix(case, 'hgh'))


def _rmmdiis_inputs(case, seed, dt):
    """A step in mid-SCF: orthonormal-looking bands, their projections, and
    the eigenvalues and eigenvectors the dense solver returned (close to the
    identity)."""
    nb = case['bands']
    psi = _waves(case, seed)
    psi = psi / (psi.square().sum((1, 2, 3), keepdim=True) * H**3).sqrt()
    v = -0.3 + 0.1 * _waves({**case, 'bands': 1, 'nk': 1}, seed, 2)[0]
    rng = np.random.default_rng(seed)
    q, r = np.linalg.qr(np.eye(nb) + 0.05 / sqrt(nb) * rng.standard_normal((nb, nb)))
    V = torch.from_numpy(q * np.sign(np.diag(r))).cuda()
    eps = torch.linspace(-0.4, 0.3, nb, dtype=torch.float64, device='cuda')
    P = 0.1 * torch.from_numpy(rng.standard_normal((nb, 8 * case['atoms']))).cuda()
    f = torch.where(torch.arange(nb, device='cuda') < 0.8 * nb, 2.0, 0.0).to(torch.float64)
    return psi.to(dt), v, eps, V, P, f, (f > 0).to(torch.float64)


def run(s):
    if s.kind == 'kinetic':
        if s.v is None:
            return s.op.apply(s.x, s.y, s.phases)
        return s.op.apply_potential(s.x, s.y, s.v, s.phases)
    if s.kind == 'vcycle':
        return s.pc(s.R, s.kpt)
    if s.kind == 'transfer':
        return s.up.apply(s.n), s.down.apply(s.v)
    if s.kind == 'residual':
        from gpaw_b200.bandops import band_combine
        P = s.pt.integrate(s.psi, {})
        R = torch.empty_like(s.psi)
        band_combine(R, s.coef, [s.Hpsi, s.psi])
        s.pt.add_M(R, P @ s.dH)
        return P, R
    if s.kind == 'xc':
        v, e = torch.zeros_like(s.n), s.gd.empty()
        E = s.xc.calculate(s.gd, s.n, v, e)
        return E, v, e
    if s.kind == 'rmmdiis':
        from gpaw_b200.wavefunctions import KPoint
        kpt = KPoint(s.psi)
        kpt.P_nM, kpt._f_t = s.P, s.f
        Hnn, Ht = s.es.subspace_matrix(s.ham, s.wfs, kpt)
        s.es.subspace_rotate(s.wfs, kpt, s.eps, s.V, Ht)
        error = s.es.update_bands(s.ham, s.wfs, kpt, s.w)
        s.wfs.orthonormalize(kpt)
        nt = s.gd.zeros()
        s.wfs.add_to_density(nt, kpt)
        return Hnn, error, kpt.psit_nG, kpt.P_nM, nt
    if s.kind == 'fold':
        return s.folded.forward(s.R)
    out = s.net.forward(s.R, keep=True)
    loss, g = s.net.loss_and_grad(out, s.T)
    return loss, out, s.net.backward(g)


# ---------------------------------------------------------------- costs

def work(case):
    kind = case['kind']
    pts = float(np.prod(_points(case)))
    z = torch.empty(0, dtype=_dtype(case)).element_size()
    rows, c = _rows(case), 2 if _dtype(case).is_complex else 1
    if kind == 'kinetic':
        v = pts * z / c if case['potential'] else 0
        return {'bytes': 2 * rows * pts * z + v, 'flops': rows * pts * c * 38}
    if kind == 'vcycle':
        # the fine stencil, two 7-point ones on 1/8 and one on 1/64 of the
        # points, the transfers and the updates
        return {'bytes': 2 * rows * pts * z, 'flops': rows * pts * c * 60}
    if kind == 'transfer':
        fine = float(np.prod([2 * n - (0 if _pbc(case) else 1) for n in _n(case)]))
        return {'bytes': 16 * case['grids'] * (pts + fine), 'flops': case['grids'] * fine * 2 * 20}
    if kind == 'residual':
        # read psi and H psi, write the residual; the functions' values are
        # counted as arithmetic on the points they cover
        m, vol = sum(2 * l + 1 for l, _, _ in _radials(case['functions'])), 0.0
        for l, rc, _ in _radials(case['functions']):
            vol += (2 * l + 1) * 4 / 3 * pi * rc**3 / H**3
        return {'bytes': 3 * rows * pts * z + 2 * rows * m * case['atoms'] * z,
                'flops': rows * (4 * case['atoms'] * vol + 3 * pts)}
    if kind == 'xc':
        return {'bytes': 8 * pts * (2 * case['spins'] + 1), 'flops': pts * 200 * case['spins']}
    if kind == 'rmmdiis':
        # bands in and out once; H_nn, S_nn and three rotations, two
        # applications of H, three preconditionings, two projections and adds
        proj = 8 * case['atoms'] * 4 / 3 * pi * 4.3**3 / H**3
        return {'bytes': 2 * rows * pts * z,
                'flops': 5 * 2.0 * rows**2 * pts + rows * pts * (3 * 38 + 3 * 60 + 40) + rows * 6 * 2 * proj}
    if kind == 'fold':
        return {'bytes': 2 * rows * pts * 4,
                'flops': 2 * rows * (pts * 30 + pts / 8 * 180 + pts / 64 * (2000 + 27 * 256))}
    conv = 27 * (2 * pts + 32 * pts / 8 + 256 * pts / 64)
    return {'bytes': 2 * rows * pts * 4, 'flops': 3 * 2 * rows * conv}


def tolerance(case):
    # about four times the errors seen against exact() over 50 cases
    f32 = case.get('dtype', 'f64') in ('f32', 'c64')
    kind = case['kind']
    if kind == 'kinetic':
        return {'rel': 4e-7 if f32 else 1.5e-15}
    if kind == 'vcycle':
        return {'rel': 3e-7 if f32 else 3e-15}
    if kind == 'transfer':
        return {'rel': 1e-15}
    if kind == 'residual':
        return {'rel': 7e-7 if f32 else 1e-14}
    if kind == 'xc':
        return {'rel': 4e-12}
    if kind == 'rmmdiis':
        return {'rel': 5e-5 if f32 else 1e-12}
    return {'rel': 2e-6 if kind == 'fold' else 8e-6}


# ---------------------------------------------------------------- 64-bit results

def _shift(x, k, axis, pbc, phase=None):
    """x at index + k along axis: wrapped (with the Bloch phase of the side it
    wraps over) or zero."""
    if k == 0:
        return x
    y = torch.roll(x, -k, axis)
    d = 0 if k > 0 else 1
    lo, m = (x.shape[axis] - k, k) if k > 0 else (0, -k)
    if not pbc:
        y.narrow(axis, lo, m).zero_()
    elif phase is not None:
        y.narrow(axis, lo, m).mul_(phase[..., d])
    return y


def _axis_phases(ph, rows):
    """Phases (nk, 3, 2) -> per axis a (rows, 1, 1, 1, 2) tensor."""
    if ph is None:
        return [None] * 3
    p = torch.from_numpy(np.asarray(ph).reshape(-1, 3, 2)).cuda()
    p = p.repeat_interleave(rows // len(p), 0)
    return [p[:, c].reshape(-1, 1, 1, 1, 2) for c in range(3)]


def _laplace(x, n, h, pbc, scale, ph=(None, None, None)):
    """scale * nabla^2 of order 2n on a grid of spacing h."""
    y = torch.zeros_like(x)
    for c in range(3):
        for k in range(-n, n + 1):
            y += scale * W2[n][abs(k)] / h**2 * _shift(x, k, x.ndim - 3 + c, pbc, ph[c])
    return y


def _restrict(x, nn, pbc, ph=(None, None, None)):
    for c in range(3):
        ax = x.ndim - 3 + c
        y = x.clone()
        for j, w in enumerate(MID[nn]):
            k = 2 * j + 1
            y += w * (_shift(x, k, ax, pbc, ph[c]) + _shift(x, -k, ax, pbc, ph[c]))
        first = 0 if pbc else 1
        x = 0.5 * y.index_select(ax, torch.arange(first, x.shape[ax], 2, device=x.device))
    return x


def _interpolate(x, nn, pbc, ph=(None, None, None)):
    for c in range(3):
        ax = x.ndim - 3 + c
        n = x.shape[ax]
        if not pbc:       # put the boundary point back in front
            x = torch.cat([torch.zeros_like(x.narrow(ax, 0, 1)), x], ax)
            n += 1
        odd = 0
        for j, w in enumerate(MID[nn]):
            odd = odd + w * (_shift(x, -j, ax, pbc, ph[c]) + _shift(x, j + 1, ax, pbc, ph[c]))
        x = torch.stack([x, odd], ax + 1).flatten(ax, ax + 1)
        if not pbc:
            x = x.narrow(ax, 1, 2 * n - 1)
    return x


def _vcycle(R, pbc, ph=(None, None, None)):
    """The three-level V-cycle: restrict -R, smooth, correct from the coarser
    grid, smooth again, interpolate, smooth on the fine grid."""
    step = 0.66666666 / (3 * -0.5 * W2[3][0] / H**2)
    K = lambda x, n, h: _laplace(x, n, h, pbc, -0.5, ph)
    r1 = _restrict(-R, 1, pbc, ph)
    d1 = 4 * step * r1
    r2 = _restrict(K(d1, 1, 2 * H) - r1, 1, pbc, ph)
    d2 = 16 * step * r2
    d2 = d2 - 16 * step * (K(d2, 1, 4 * H) - r2)
    d1 = d1 - _interpolate(d2, 1, pbc, ph)
    d1 = d1 - 4 * step * (K(d1, 1, 2 * H) - r1)
    d0 = _interpolate(-d1, 1, pbc, ph)
    return step * (K(d0, 3, H) - R) - d0


def _spline(f, dr, r):
    """The cubic spline through the table f (spacing dr) with zero slope at
    both ends, at the radii r."""
    n = len(f) - 1
    A = 4.0 * np.eye(n + 1) + np.eye(n + 1, k=1) + np.eye(n + 1, k=-1)
    A[0, 0] = A[n, n] = 2.0
    b = np.zeros(n + 1)
    b[1:n] = f[2:] - 2 * f[1:n] + f[:n - 1]
    b[0], b[n] = f[1] - f[0], f[n - 1] - f[n]
    m = torch.from_numpy(np.linalg.solve(A, 6.0 / dr**2 * b)).cuda()      # second derivatives
    f = torch.from_numpy(f).cuda()
    i = (r / dr).long().clamp_(0, n - 1)
    u = r - i.to(torch.float64) * dr
    s1 = (f[i + 1] - f[i]) / dr - (m[i] / 3 + m[i + 1] / 6) * dr
    return f[i] + u * (s1 + u * (0.5 * m[i] + u * (m[i + 1] - m[i]) / (6 * dr)))


def _harmonics(l, x, y, z):
    if l == 0:
        return [torch.full_like(x, 1 / sqrt(4 * pi))]
    if l == 1:
        c = sqrt(3 / (4 * pi))
        return [c * y, c * z, c * x]
    c, c0 = sqrt(15 / (4 * pi)), sqrt(5 / (16 * pi))
    return [c * x * y, c * y * z, c0 * (2 * z * z - x * x - y * y), c * x * z,
            0.5 * c * (x * x - y * y)]


def _functions(case, seed, functions):
    """Every localized function on the grid: (functions, points)."""
    n, N = _points(case), _n(case)
    out = []
    for spos in _atoms(case, seed):
        d = []
        for c in range(3):
            x = torch.arange(n[c], device='cuda', dtype=torch.float64) + (0 if _pbc(case) else 1)
            x = x * H - spos[c] * N[c] * H
            L = N[c] * H
            d.append(x - L * torch.round(x / L) if _pbc(case) else x)
        x, y, z = (t.contiguous() for t in torch.broadcast_tensors(
            d[0][:, None, None], d[1][None, :, None], d[2][None, None, :]))
        r = (x * x + y * y + z * z).sqrt()
        for l, rc, f in _radials(functions):
            inside = r < rc
            g = torch.zeros_like(r)
            g[inside] = _spline(f, rc / (len(f) - 1), r[inside])
            out.extend((g * Y).reshape(-1) for Y in _harmonics(l, x, y, z))
    return torch.stack(out)


def _pbe(n, sig):
    """Energy per volume of PBE for spin densities n (2, G) and sigma
    (3, G) = (uu, ud, dd)."""
    kappa, beta, gam = 0.804, 0.066725, 0.031091
    mu = beta * pi**2 / 3

    def ex(n, a2):
        rs = (3 / (4 * pi) / n)**(1 / 3)
        s2 = a2 * (rs / ((18 * pi)**(1 / 3) * n))**2
        e = -9 / (8 * pi) * (2 * pi / 3)**(1 / 3) / rs
        return n * e * (1 + kappa - kappa / (1 + mu * s2 / kappa))

    def G(t, A, a1, b1, b2, b3, b4):
        return -2 * A * (1 + a1 * t * t) * torch.log1p(
            1 / (2 * A * t * (b1 + t * (b2 + t * (b3 + t * b4)))))

    e = 0.5 * (ex(2 * n[0], 4 * sig[0]) + ex(2 * n[1], 4 * sig[2]))
    nt = n[0] + n[1]
    a2 = sig[0] + 2 * sig[1] + sig[2]
    zeta = (n[0] - n[1]) / nt
    rs = (3 / (4 * pi) / nt)**(1 / 3)
    t = rs.sqrt()
    e0 = G(t, gam, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294)
    e1 = G(t, 0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    al = -G(t, 0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    c1 = 1 / (2**(4 / 3) - 2)
    f = c1 * ((1 + zeta)**(4 / 3) + (1 - zeta)**(4 / 3) - 2)
    ec = e0 + al * f * (1 - zeta**4) * 9 / (8 * c1) + (e1 - e0) * f * zeta**4
    phi = 0.5 * ((1 + zeta)**(2 / 3) + (1 - zeta)**(2 / 3))
    t2 = pi * (4 / (9 * pi))**(1 / 3) / 16 * a2 * rs / (nt * phi)**2
    A = beta / (gam * torch.expm1(-ec / (gam * phi**3)))
    num = 1 + A * t2
    Hc = gam * phi**3 * torch.log1p(beta / gam * t2 * num / (num + (A * t2)**2))
    return e + nt * (ec + Hc)


def _gradient(x, c, h, pbc):
    ax = x.ndim - 3 + c
    y = torch.zeros_like(x)
    for k, w in ((1, 2 / 3), (2, -1 / 12)):
        y += w / h * (_shift(x, k, ax, pbc) - _shift(x, -k, ax, pbc))
    return y


def _exact_xc(case, seed):
    n, pbc, h = _density(case, seed), _pbc(case), H / 2
    ns = len(n)
    g = [_gradient(n, c, h, pbc) for c in range(3)]
    pair = [(0, 0)] if ns == 1 else [(0, 0), (0, 1), (1, 1)]
    sig = torch.stack([sum(gc[a] * gc[b] for gc in g) for a, b in pair])
    e = torch.empty_like(n[0])
    v, ds = torch.empty_like(n), torch.empty_like(sig)
    floor = 1e-10 / ns
    for k in range(len(e)):          # plane by plane: the graph of the derivatives is large
        nk = n[:, k].clamp_min(floor).requires_grad_()
        sk = sig[:, k].clone().requires_grad_()
        if ns == 1:
            ek = _pbe(torch.stack([nk[0] / 2] * 2), torch.stack([sk[0] / 4] * 3))
        else:
            ek = _pbe(nk, sk)
        v[:, k], ds[:, k] = torch.autograd.grad(ek.sum(), [nk, sk])
        e[k] = ek.detach()
    for c in range(3):
        for s in range(ns):
            flux = 2 * ds[2 * s] * g[c][s]
            if ns == 2:
                flux = flux + ds[1] * g[c][1 - s]
            v[s] -= _gradient(flux, c, h, pbc)
    return float(e.sum() * h**3), v, e


def _exact_rmmdiis(case, seed):
    dt, pbc = _dtype(case), _pbc(case)
    psi, v, eps, V, P, f, w = _rmmdiis_inputs(case, seed, dt)
    real = lambda t: t.to(dt).to(torch.float64)
    psi, v, P = psi.to(torch.float64), real(v), real(P)
    phi, dv = _functions(case, seed, 'hgh'), H**3
    dH = _dh_matrix(case, 'hgh')
    T = lambda x: _laplace(x, 3, H, pbc, -0.5) + v * x
    flat = lambda x: x.reshape(len(x), -1)
    project = lambda x: dv * flat(x) @ phi.T
    dot = lambda a, b: (flat(a) * flat(b)).sum(1) * dv
    col = lambda a: a.reshape(-1, 1, 1, 1)

    def residual(x, Tx, Px):
        return Tx - col(eps) * x + (Px @ dH.T @ phi).reshape(x.shape)

    Ht = T(psi)
    Hnn = dv * flat(psi) @ flat(Ht).T + P @ dH @ P.T
    Hnn = 0.5 * (Hnn + Hnn.T)
    rot = lambda x: (V.T @ flat(x)).reshape(x.shape)
    psi, P = rot(psi), V.T @ P
    R = [residual(psi, rot(Ht), P)]
    error = (w * dot(R[0], R[0])).sum()
    d = _vcycle(R[0], pbc)
    dR = residual(d, T(d), project(d))
    lam = -dot(dR, R[0]) / dot(dR, dR)
    xs = [psi, psi + col(lam) * d]
    R.append(R[0] + col(lam) * dR)
    nxt = xs[1] + col(lam) * _vcycle(R[1], pbc)
    xs.append(nxt)
    R.append(residual(nxt, T(nxt), project(nxt)))
    A = -torch.ones((len(psi), 4, 4), dtype=torch.float64, device='cuda')
    for i in range(3):
        for j in range(3):
            A[:, i, j] = dot(R[i], R[j])
    A[:, 3, 3] = 0.0
    b = torch.zeros((len(psi), 4), dtype=torch.float64, device='cuda')
    b[:, 3] = -1.0
    al = torch.linalg.solve(A, b)
    x = sum(col(al[:, i]) * xs[i] for i in range(3))
    x = x + 0.1 * _vcycle(sum(col(al[:, i]) * R[i] for i in range(3)), pbc)
    L = torch.linalg.cholesky(dv * flat(x) @ flat(x).T)
    x = torch.linalg.solve_triangular(L, flat(x), upper=False).reshape(x.shape)
    return Hnn, error, x, project(x), (col(f) * x.square()).sum(0)


def _conv(x, w, pbc):
    w = w.reshape(*w.shape[:2], 3, 3, 3)
    x = F.pad(x, (1,) * 6, mode='circular') if pbc else F.pad(x, (1,) * 6)
    return F.conv3d(x, w)


def _exact_net(case, seed):
    pbc, train = _pbc(case), case['kind'] == 'train'
    shape = (_rows(case), *_points(case))
    R = _randn(shape, seed, torch.float32).to(torch.float64)
    scale = 1.0 if train else 0.05
    p = {k: (w * (scale if k in ('w0', 'wp') else 1.0)).bfloat16().double().requires_grad_(train)
         for k, w in _params(seed).items()}
    s = R.square().mean((1, 2, 3), keepdim=True).sqrt() if train else 1.0
    x = (R / s)[:, None]
    a1 = _conv(_restrict(x, 1, pbc), p['wa'], pbc)
    a2 = _conv(_restrict(a1, 1, pbc), p['wb'], pbc)
    b1 = _conv(_interpolate(a2, 1, pbc) + a1, p['wc'], pbc)
    y = _conv(_interpolate(b1, 1, pbc), p['wp'], pbc) + _conv(x, p['w0'], pbc)
    y = y[:, 0] * s
    if not train:
        return y
    T = _randn(shape, seed, torch.float32, 1).to(torch.float64)
    K = lambda u: _laplace(u, 1, H, pbc, -0.5) + u
    loss = (K(y - T).square().sum((1, 2, 3)) / K(T).square().sum((1, 2, 3))).mean()
    names = list(p)
    return float(loss.detach()), y.detach(), dict(zip(names, torch.autograd.grad(loss, [p[k] for k in names])))


def exact(case, seed):
    kind, pbc = case['kind'], _pbc(case)
    shape, dt = (_rows(case), *_points(case)), _dtype(case)
    wide = torch.complex128 if dt.is_complex else torch.float64
    if kind == 'kinetic':
        ph = _axis_phases(_phases(case, seed), shape[0])
        x = _randn(shape, seed, dt).to(wide)
        y = _laplace(x, 3, H, pbc, -0.5, ph)
        if case['potential']:
            single = dt in (torch.float32, torch.complex64)
            v = _randn(shape[1:], seed, torch.float64, 1)
            y += (v.float().double() if single else v) * x
        return y
    if kind == 'vcycle':
        return _vcycle(_randn(shape, seed, dt).to(wide), pbc, _axis_phases(_phases(case, seed), shape[0]))
    if kind == 'transfer':
        n = torch.cat([_density(case, seed + i) for i in range(case['grids'])])
        fine = [2 * m - (0 if pbc else 1) for m in _n(case)]
        return _interpolate(n, 3, pbc), _restrict(_randn((case['grids'], *fine), seed), 3, pbc)
    if kind == 'residual':
        phi = _functions(case, seed, case['functions'])
        psi, Hpsi = (_waves(case, seed, i).to(dt).to(torch.float64).flatten(1) for i in (0, 1))
        e = torch.linspace(-0.4, 0.3, shape[0], dtype=torch.float64, device='cuda')[:, None]
        P = H**3 * psi @ phi.T
        R = Hpsi - e * psi + P @ _dh_matrix(case, case['functions']).to(dt).double() @ phi
        return P, R.reshape(shape)
    if kind == 'xc':
        return _exact_xc(case, seed)
    if kind == 'rmmdiis':
        return _exact_rmmdiis(case, seed)
    return _exact_net(case, seed)
