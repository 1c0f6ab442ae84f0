"""GPU: the kernels that a rule on size, type or alignment chooses, at the
sizes where their tiles and remainders can go wrong, against the oracle.

Tolerances: FP64 1e-12 and FP32 1e-5 norm-wise, as in the other kernel tests;
weight gradients 3e-6 of the sum of the absolute products: FP32 sums of N
terms as 32 or more partial sums err by at most a few N/32 ulp of that sum,
and N / 32 < 20 rounding steps here."""
import numpy as np
import pytest
import torch

from conftest import bloch_phases, relerr
from oracle import fd

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-12, torch.complex128: 1e-12,
       torch.float32: 1e-5, torch.complex64: 1e-5}


ROWS = [((24, 75, 75), (0, 0, 0), 48),   # a last row tile of few rows
        ((20, 26, 77), (1, 0, 1), 100),  # one tile, wrapped halo columns
        ((20, 29, 101), (0, 1, 0), 80),  # rows of more than three warps, wrapped halo rows
        ((17, 36, 75), (1, 1, 1), 96)]   # everything wrapped


@pytest.mark.parametrize('n_c,pbc,nb', ROWS + [
    ((31, 31, 31), (0, 0, 0), 48),       # rows too short for the row kernel's copies
    ((24, 75, 75), (0, 0, 0), 32),
    ((40, 7, 33), (1, 0, 1), 80),
    ((20, 29, 98), (0, 1, 0), 64),
    ((17, 36, 21), (1, 1, 1), 96),
])
@pytest.mark.parametrize('dtype', [torch.float64, torch.float32, torch.complex128,
                                   torch.complex64])
@pytest.mark.parametrize('kind', ['laplace3', 'laplace1', 'gradient'])
def test_row_stencil(n_c, pbc, nb, dtype, kind):
    """Every band of apply equals the result on that band alone (a call so
    small that it marches), three bands equal the oracle, and the potential is
    added (k-point batches of phases for complex data).  The batches of ROWS
    take the row kernel, but for 7-point FP32 stencils, which march, and
    complex128 without phases, whose rows suit the TMA kernel."""
    from gpaw_b200.fd_operators import Gradient, Laplace
    from gpaw_b200.grid_descriptor import GridDescriptor
    N = np.array(n_c) + (1 - np.array(pbc))
    gd = GridDescriptor(N, 0.3 * N, pbc)
    c = complex if dtype.is_complex else float
    op = Gradient(gd, 1, 1.0, 2, c) if kind == 'gradient' else Laplace(gd, -0.5, int(kind[-1]), c)
    g = torch.Generator(device='cuda').manual_seed(3)
    x = torch.randn((nb,) + n_c, generator=g, device='cuda', dtype=dtype)
    real = torch.float32 if dtype in (torch.float32, torch.complex64) else torch.float64
    v = torch.randn(n_c, generator=g, device='cuda', dtype=real)
    ks = [(0.13, -0.21, 0.37), (0.4, 0.1, -0.3)]
    ph = np.array([bloch_phases(pbc, k) for k in ks]) if dtype.is_complex else None
    y, yv = torch.empty_like(x), torch.empty_like(x)
    if (n_c, pbc, nb) in ROWS:
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            op.apply(x, y, ph)
            torch.cuda.synchronize()
        want = 'march_star_kernel' if kind == 'laplace1' and dtype == torch.float32 else \
               'star_tma_kernel' if dtype == torch.complex128 and not any(pbc) else 'rows_star_kernel'
        assert any(want in e.key for e in prof.key_averages())
    op.apply(x, y, ph)
    op.apply_potential(x, yv, v, ph)
    wide = np.complex128 if dtype.is_complex else np.float64
    for b in (0, nb // 2 - 1, nb - 1):
        p = None if ph is None else ph[b // (nb // 2)]
        h = x[b].cpu().numpy().astype(wide)[None]
        ref = fd.fd_apply(op.coef_p, op.offset_pc, h, pbc, p)
        assert relerr(y[b:b + 1].cpu().numpy(), ref) < TOL[dtype]
        ref = ref + v.cpu().numpy().astype(np.float64) * h
        assert relerr(yv[b:b + 1].cpu().numpy(), ref) < TOL[dtype]
    one = torch.empty_like(x[:1])
    for b in range(nb):
        op.apply(x[b:b + 1], one, None if ph is None else ph[b // (nb // 2)])
        assert torch.equal(y[b:b + 1], one)


@pytest.mark.parametrize('N,pbc', [((44, 36, 76), (0, 0, 0)), ((20, 44, 36), (1, 0, 1)),
                                   ((28, 20, 140), (0, 1, 0))])
@pytest.mark.parametrize('nn', [1, 3])
@pytest.mark.parametrize('dtype', [torch.float64, torch.complex64])
def test_transfer_tiles(N, pbc, nn, dtype):
    """Transfers whose tiles end inside the grid, mixed boundaries, a batch of
    phases, and the y epilogue of the interpolation."""
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.transformers import Transformer
    gf = GridDescriptor(N, 0.3 * np.array(N), pbc)
    gc = gf.coarsen()
    c = complex if dtype.is_complex else float
    ks = [(0.13, -0.21, 0.37), (0.4, 0.1, -0.3)]
    ph = np.array([bloch_phases(pbc, k) for k in ks]) if dtype.is_complex else None
    g = torch.Generator(device='cuda').manual_seed(5)
    for gi, go in ((gf, gc), (gc, gf)):
        t = Transformer(gi, go, nn, c)
        x = torch.randn((6,) + tuple(gi.n_c), generator=g, device='cuda', dtype=dtype)
        y = t.apply(x, None, ph)
        wide = np.complex128 if dtype.is_complex else np.float64
        h = x.cpu().numpy().astype(wide)
        ot = fd.Transformer(*[fd.Grid(d.N_c, d.cell_cv, d.pbc_c) for d in (gi, go)], nn)
        ref = np.concatenate([ot.apply(h[3 * k:3 * k + 3], None if ph is None else ph[k])
                              for k in range(2)])
        assert relerr(y.cpu().numpy(), ref) < TOL[dtype]
        if gi is gc and ph is None:
            z = torch.randn(y.shape, generator=g, device='cuda', dtype=dtype)
            o = torch.empty_like(z)
            t.apply_axpy(x, o, -0.7, z, 0.3)
            assert relerr(o.cpu().numpy(), -0.7 * ref + 0.3 * z.cpu().numpy()) < TOL[dtype]


@pytest.mark.parametrize('pbc', [(1, 0, 1), (0, 1, 0)])
@pytest.mark.parametrize('nspins,stencil', [(1, 1), (1, 3), (2, 2), (2, 4)])
def test_gga_two_launches(pbc, nspins, stencil):
    """The fused gradient / functional / divergence form against the separate
    launches it replaces on axis-aligned grids (mixed boundaries, radii 1-4)."""
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.xc import XC
    N = np.array((18, 23, 37))
    gd = GridDescriptor(N, 0.4 * N, pbc)
    g = torch.Generator(device='cuda').manual_seed(1)
    n = torch.rand((nspins,) + tuple(gd.n_c), generator=g, device='cuda', dtype=torch.float64) + 0.1
    out = []
    for fused in (True, False):
        xc = XC('PBE', stencil=stencil)
        xc.set_grid_descriptor(gd)
        assert xc.on_axes
        xc.on_axes = fused
        v, e = torch.full_like(n, 0.25), gd.empty()
        xc.calculate(gd, n, v, e)
        out.append((v.cpu().numpy(), e.cpu().numpy()))
    assert relerr(out[0][0], out[1][0]) < 1e-12
    assert relerr(out[0][1], out[1][1]) < 1e-13


@pytest.mark.parametrize('n_c,pbc,nb', [((15, 9, 33), (0, 0, 0), 2), ((28, 28, 28), (1, 1, 1), 3),
                                        ((5, 4, 6), (1, 0, 1), 1)])
@pytest.mark.parametrize('cin,cout', [(1, 1), (16, 1), (1, 16), (16, 16), (2, 3)])
def test_weight_gradient(n_c, pbc, nb, cin, cout):
    import ctypes
    from gpaw_b200 import _native as nat
    from oracle import learned as ol
    g = torch.Generator(device='cuda').manual_seed(2)
    x = torch.randn((nb, cin) + n_c, generator=g, device='cuda', dtype=torch.float32)
    dy = torch.randn((nb, cout) + n_c, generator=g, device='cuda', dtype=torch.float32)
    dw = torch.ones((cout, cin, 27), device='cuda')
    nat.check(nat.lib().gb_conv3d_backward_weight(
        nat.ptr(x), nat.ptr(dy), nat.ptr(dw), nb, cin, cout, nat.i64(n_c),
        (ctypes.c_int * 3)(*pbc), nat.stream_of(x)), 'gb_conv3d_backward_weight')
    h = [t.double().cpu().numpy() for t in (x, dy)]
    ref = 1.0 + ol.conv_bwd_w(*h, pbc)
    bound = 1.0 + ol.conv_bwd_w(*[np.abs(t) for t in h], pbc)
    assert (np.abs(dw.cpu().numpy() - ref) < 3e-6 * bound).all()


@pytest.mark.parametrize('nx', [1, 16, 33, 81, 170])
@pytest.mark.parametrize('ls', [(0,), (0, 1, 2), (0, 1, 0, 1, 0, 2)])
@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_lfc_tensor_cores(nx, ls, dtype):
    """add and integrate of 1, 9 and 14 functions per atom on a zero-boundary
    grid whose point count is no multiple of 4 or 8, with band counts around
    the 16-band tiles; points outside every sphere keep their bits, and a
    band's result does not depend on the others."""
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.lfc import LFC
    from gpaw_b200.spline import Spline
    from oracle import lfc as ol
    N = np.array((16, 18, 14))
    rc = 2.1
    r = np.linspace(0, rc, 41)
    spl = [(l, rc, np.exp(-r**2) * (1 + 0.3 * j)) for j, l in enumerate(ls)]
    gd = GridDescriptor(N, 0.4 * N, False)
    spos = 0.25 + 0.5 * np.random.default_rng(4).random((3, 3))
    lfc = LFC(gd, [[Spline.from_data(*s) for s in spl]] * 3, cut=True)
    lfc.set_positions(spos)
    Phi = ol.dense_functions(gd.N_c, gd.cell_cv, gd.pbc_c, spos, [spl] * 3)
    g = torch.Generator(device='cuda').manual_seed(nx)
    a = torch.randn((nx,) + tuple(gd.n_c), generator=g, device='cuda', dtype=dtype)
    c = torch.randn((nx, lfc.Mmax), generator=g, device='cuda', dtype=dtype)
    P = lfc.integrate(a, {})
    assert relerr(P.double().cpu().numpy(), ol.integrate(a.double().cpu().numpy(), Phi, gd.dv)) < TOL[dtype]
    b = a.clone()
    lfc.add_M(b, c)
    assert relerr(b.double().cpu().numpy(),
                  ol.add(a.double().cpu().numpy(), c.double().cpu().numpy(), Phi)) < TOL[dtype]
    bare = torch.from_numpy(~np.any(Phi.reshape(lfc.Mmax, -1) != 0, axis=0)).cuda()
    assert bare.any() and torch.equal(b.flatten(1)[:, bare], a.flatten(1)[:, bare])
    k = max(0, nx - 2)
    assert torch.equal(lfc.integrate(a[k:].contiguous(), {}), P[k:])
    one = a[k:].clone()
    lfc.add_M(one, c[k:].contiguous())
    assert torch.equal(one, b[k:])


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_potential_of_a_skew_cell(dtype):
    """The potential joins stencils with points off the axes as it does the others."""
    from gpaw_b200.fd_operators import Laplace
    from gpaw_b200.grid_descriptor import GridDescriptor
    gd = GridDescriptor((12, 10, 14), [[4.0, 0, 0], [1.5, 4.0, 0], [0.5, 0.7, 4.5]], True)
    lap = Laplace(gd, -0.5, 2)
    assert not lap.cfd
    g = torch.Generator(device='cuda').manual_seed(7)
    x = torch.randn((3,) + tuple(gd.n_c), generator=g, device='cuda', dtype=dtype)
    v = torch.randn(tuple(gd.n_c), generator=g, device='cuda', dtype=dtype)
    y = torch.empty_like(x)
    lap.apply_potential(x, y, v)
    h = x.cpu().numpy().astype(np.float64)
    ref = fd.fd_apply(lap.coef_p, lap.offset_pc, h, (1, 1, 1)) + v.cpu().numpy().astype(np.float64) * h
    assert relerr(y.cpu().numpy(), ref) < TOL[dtype]
