"""GPU: which kernel a call takes, for the forms whose rule was drawn by
measuring both sides, and what a rule must not change: a band's result must
not depend on how many bands come with it."""
import numpy as np
import pytest
import torch

from conftest import bloch_phases, relerr
from oracle import fd

pytestmark = pytest.mark.gpu


def kernels(f):
    """Names of the kernels f() launches."""
    f()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        f()
        torch.cuda.synchronize()
    return [e.key for e in prof.key_averages()]


def stencil_on(n_c, pbc, kind, dtype):
    """Laplace(gd, -1/2, n) for kind n, the derivative along axis 1 for 'g'."""
    from gpaw_b200.fd_operators import Gradient, Laplace
    from gpaw_b200.grid_descriptor import GridDescriptor
    N = np.array(n_c) + (1 - np.array(pbc))
    gd = GridDescriptor(N, 0.3 * N, pbc)
    c = complex if dtype.is_complex else float
    return Gradient(gd, 1, 1.0, 3, c) if kind == 'g' else Laplace(gd, -0.5, kind, c)


def phases_of(pbc, dtype, k=(0.13, -0.21, 0.37)):
    return bloch_phases(pbc, k) if dtype.is_complex else None


def randn(shape, dtype, seed=1):
    g = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn(shape, generator=g, device='cuda', dtype=dtype)


@pytest.mark.parametrize('n_c,pbc,nb', [((24, 75, 75), (0, 0, 0), 48), ((30, 40, 77), (1, 1, 1), 48)])
@pytest.mark.parametrize('kind', [1, 2, 3, 4, 'g'])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64, torch.complex64])
def test_stencil_of_one_band_and_of_many(n_c, pbc, nb, kind, dtype):
    """Odd rows: a batch takes the row kernel, a band alone the marching one,
    and both give it the same bits."""
    op = stencil_on(n_c, pbc, kind, dtype)
    ph = phases_of(pbc, dtype)
    x = randn((nb,) + n_c, dtype)
    y, one = torch.empty_like(x), torch.empty_like(x[:1])
    names = kernels(lambda: op.apply(x, y, ph))
    rows = not (kind == 1 and dtype == torch.float32)
    assert any(('rows_star_kernel' if rows else 'march_star_kernel') in k for k in names), names
    assert any('march_star_kernel' in k for k in kernels(lambda: op.apply(x[:1], one, ph)))
    for b in (0, nb // 2, nb - 1):
        op.apply(x[b:b + 1], one, ph)
        assert torch.equal(one, y[b:b + 1])


@pytest.mark.parametrize('kind', [1, 2, 3, 4, 'g'])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64, torch.complex64, torch.complex128])
def test_plain_stencils_carry_no_epilogue(kind, dtype):
    """apply() runs a kernel without the general epilogue (last template
    argument below 2), whatever the radius; a potential is added all the same."""
    n_c, pbc = (20, 24, 32), (1, 0, 1)
    op = stencil_on(n_c, pbc, kind, dtype)
    ph = np.ones((3, 2), complex) if dtype.is_complex else None
    x = randn((3,) + n_c, dtype)
    y, z = torch.empty_like(x), torch.empty_like(x)
    names = [k for k in kernels(lambda: op.apply(x, y, ph)) if 'star_tma_kernel' in k]
    assert names and not any(', 2>' in k for k in names), names
    v = randn(n_c, x.real.dtype if dtype.is_complex else dtype, 2)
    op.apply_potential(x, z, v, ph)
    tol = 1e-12 if dtype in (torch.float64, torch.complex128) else 1e-5
    assert (z - (y + v * x)).abs().max() < tol * y.abs().max()


@pytest.mark.parametrize('n,pbc,kind,dtype', [(15, 0, 1, torch.float64), (19, 1, 1, torch.float64),
                                              (25, 0, 4, torch.float64), (25, 1, 2, torch.complex64),
                                              (27, 0, 4, torch.float32)])
def test_short_rows_march(n, pbc, kind, dtype):
    """Rows of fewer than 28 elements do not fill the row kernel's CTAs
    (coarse multigrid levels), however many bands there are."""
    op = stencil_on((n, n, n), (pbc,) * 3, kind, dtype)
    ph = phases_of((pbc,) * 3, dtype)
    x = randn((240, n, n, n), dtype)
    y, one = torch.empty_like(x), torch.empty_like(x[:1])
    assert any('march_star_kernel' in k for k in kernels(lambda: op.apply(x, y, ph)))
    op.apply(x[77:78], one, ph)
    assert torch.equal(one, y[77:78])


@pytest.mark.parametrize('n_c,pbc,nb,kind,dtype,kernel', [
    ((56, 56, 56), (1, 1, 1), 60, 6, torch.float64, 'rows'),      # radius 5 and 6
    ((45, 52, 61), (0, 1, 0), 60, 6, torch.float32, 'rows'),
    ((40, 47, 50), (1, 1, 1), 60, 5, torch.complex64, 'rows'),
    ((40, 41, 43), (1, 0, 1), 60, 6, torch.complex128, 'rows'),
    ((40, 96, 96), (0, 0, 0), 30, 6, torch.float64, 'tile'),      # few rows per tile
    ((30, 40, 257), (1, 0, 1), 30, 5, torch.float64, 'tile'),
    ((24, 25, 301), (1, 1, 1), 30, 6, torch.complex64, 'tile'),
    ((20, 20, 450), (1, 1, 1), 30, 6, torch.float32, 'march'),
    ((44, 44, 44), (0, 0, 0), 60, 6, torch.complex128, 'march'),
    ((24, 24, 24), (1, 1, 1), 10, 6, torch.float64, 'march'),     # a small call
    ((30, 33, 131), (1, 1, 1), 40, 4, torch.complex128, 'tile'),  # one row per tile, wrapped
    ((30, 33, 131), (0, 0, 0), 40, 4, torch.complex128, 'march'),
    ((24, 25, 301), (0, 0, 0), 40, 3, torch.float64, 'march'),
    ((24, 25, 301), (1, 1, 1), 40, 3, torch.float64, 'rows'),
])
def test_large_radius_and_long_rows(n_c, pbc, nb, kind, dtype, kernel):
    """Radius 5 and 6 and rows of which a tile holds few: the kernel that is
    the fastest there, the oracle's values with and without a
    potential, and the bits of a band alone."""
    op = stencil_on(n_c, pbc, kind, dtype)
    ph = phases_of(pbc, dtype)
    x = randn((nb,) + n_c, dtype)
    y, z, one = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x[:1])
    names = kernels(lambda: op.apply(x, y, ph))
    assert any(f'{kernel}_star_kernel' in k for k in names), names
    v = randn(n_c, x.real.dtype if dtype.is_complex else dtype, 2)
    op.apply_potential(x, z, v, ph)
    wide = np.complex128 if dtype.is_complex else np.float64
    tol = 1e-12 if dtype in (torch.float64, torch.complex128) else 1e-5
    for b in (0, nb - 1):
        h = x[b].cpu().numpy().astype(wide)[None]
        ref = fd.fd_apply(op.coef_p, op.offset_pc, h, pbc, ph)
        assert relerr(y[b:b + 1].cpu().numpy(), ref) < tol
        assert relerr(z[b:b + 1].cpu().numpy(), ref + v.cpu().numpy() * h) < tol
    for b in (0, nb // 2):
        op.apply(x[b:b + 1], one, ph)
        assert torch.equal(one, y[b:b + 1])


def lfc_on(N, pbc, natoms, ls, seed=3):
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.lfc import LFC
    from gpaw_b200.spline import Spline
    rc = 3.4
    r = np.linspace(0, rc, 41)
    spl = [Spline.from_data(l, rc, np.exp(-(r / 1.5)**2) * (1 + 0.3 * j)) for j, l in enumerate(ls)]
    gd = GridDescriptor((N, N, N), (0.38 * N,) * 3, pbc)
    lfc = LFC(gd, [spl] * natoms, cut=True)
    lfc.set_positions(0.2 + 0.6 * np.random.default_rng(seed).random((natoms, 3)))
    return gd, lfc


@pytest.mark.parametrize('N,pbc,ls', [(24, 0, (0, 0, 1)),       # 23^3 points: no multiple of 4
                                      (24, 1, (0, 1, 2)),       # 9 functions
                                      (24, 0, (0, 1, 0, 1, 0, 2))])
@pytest.mark.parametrize('nx', [1, 2, 40])
def test_fp32_lfc_outside_the_bricks(N, pbc, ls, nx):
    """FP32 data that the bricks do not take: FP32 sums, point by point and
    group by group (widened for the FP64 matrix instructions they took up to
    four times as long), one kernel each whatever the number of bands."""
    gd, lfc = lfc_on(N, pbc, 5, ls)
    g = torch.Generator(device='cuda').manual_seed(nx)
    a = torch.randn((nx,) + tuple(gd.n_c), generator=g, device='cuda', dtype=torch.float32)
    c = torch.randn((nx, lfc.Mmax), generator=g, device='cuda', dtype=torch.float32)
    names = kernels(lambda: lfc.integrate(a, {}))
    assert any('lfc_integrate_kernel' in k for k in names) and not any('mma' in k for k in names)
    b = a.clone()
    names = kernels(lambda: lfc.add_M(b, c))
    assert any('lfc_add_bands_kernel' in k for k in names) and not any('mma' in k for k in names)
    b = a.clone()
    lfc.add_M(b, c)
    P = lfc.integrate(a, {})
    one = a[nx - 1:].clone()
    lfc.add_M(one, c[nx - 1:].contiguous())
    assert torch.equal(one, b[nx - 1:])
    assert torch.equal(lfc.integrate(a[nx - 1:].contiguous(), {}), P[nx - 1:])


@pytest.mark.parametrize('ls', [(0,), (0, 0, 1), (0, 1, 2)])
@pytest.mark.parametrize('natoms', [1, 7])
def test_fp64_lfc_of_one_grid_and_of_many(ls, natoms):
    """Projections have the same bits for a band alone, in a block of 16 and
    among 37; so has what add gives a block.  A single grid is added to by
    another kernel: each sum of up to 7 x 9 products may then round
    differently, by at most 64 ulp of the sum of their absolute values."""
    gd, lfc = lfc_on(24, 0, natoms, ls)
    g = torch.Generator(device='cuda').manual_seed(natoms)
    a = torch.randn((37,) + tuple(gd.n_c), generator=g, device='cuda', dtype=torch.float64)
    c = torch.randn((37, lfc.Mmax), generator=g, device='cuda', dtype=torch.float64)
    P, b = lfc.integrate(a, {}), a.clone()
    lfc.add_M(b, c)
    Phi = gd.zeros(lfc.Mmax)
    lfc.add_M(Phi, torch.eye(lfc.Mmax, dtype=torch.float64, device='cuda'))
    size = a.abs() + torch.einsum('xM,Mijk->xijk', c.abs(), Phi.abs())
    for x0, x1 in ((0, 1), (20, 21), (36, 37), (5, 21)):
        part = a[x0:x1].clone()
        names = kernels(lambda: lfc.integrate(part, {}))
        assert any('lfc_integrate_mma_kernel' in k for k in names)
        assert torch.equal(lfc.integrate(part, {}), P[x0:x1])
        lfc.add_M(part, c[x0:x1].contiguous())
        if x1 - x0 > 1:
            assert torch.equal(part, b[x0:x1])
        else:
            assert ((part - b[x0:x1]).abs() <= 64 * 2.3e-16 * size[x0]).all()


@pytest.mark.parametrize('nn', [2, 3, 4])
@pytest.mark.parametrize('n0,pbc', [(16, (1, 1, 1)), (20, (0, 1, 0)), (28, (1, 0, 1)), (36, (0, 0, 0))])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64, torch.complex64, torch.complex128])
def test_interpolation_takes_several_planes(nn, n0, pbc, dtype):
    """A block interpolates four coarse planes (eight in FP32), so that a
    plane is read about twice and not once per tap; plane counts around those
    blocks against the oracle."""
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.transformers import Transformer
    N = np.array((n0, 20, 44))
    gf = GridDescriptor(N, 0.3 * N, pbc)
    gc = gf.coarsen()
    t = Transformer(gc, gf, nn, complex if dtype.is_complex else float)
    ph = phases_of(pbc, dtype)
    x = randn((3,) + tuple(gc.n_c), dtype)
    names = kernels(lambda: t.apply(x, None, ph))
    planes = 8 if dtype == torch.float32 else 4
    assert any(f', {2 * nn}, {planes}, 16' in k for k in names if 'interpolate_x_kernel' in k), names
    h = x.cpu().numpy().astype(np.complex128 if dtype.is_complex else np.float64)
    ref = fd.Transformer(*[fd.Grid(d.N_c, d.cell_cv, d.pbc_c) for d in (gc, gf)], nn).apply(h, ph)
    tol = 1e-12 if dtype in (torch.float64, torch.complex128) else 1e-5
    assert relerr(t.apply(x, None, ph).cpu().numpy(), ref) < tol


def test_lfc_object_size():
    """An object of one function per atom (a local potential, an ion charge)
    keeps about 95 bytes on the device per covered point and atom: 8 + 4 of
    values, 30 of indices, 32 of padded FP32 rows, and 8-point blocks with as
    many rows as there are functions; 20 allocations may round up by 2 MB."""
    from gpaw_b200.grid_descriptor import GridDescriptor
    from gpaw_b200.lfc import LFC
    from gpaw_b200.spline import Spline
    rc = 3.6
    spl = Spline.from_data(0, rc, np.exp(-np.linspace(0, rc, 41)**2))
    gd = GridDescriptor((96, 96, 96), (96 * 0.19,) * 3, True)
    lfc = LFC(gd, [[spl]] * 40, cut=True)
    lfc.set_positions(np.random.default_rng(2).random((40, 3)))
    rows = int(lfc.lfc.ngm.sum())
    del lfc.lfc
    lfc.my_atom_indices = None
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    lfc.set_positions(np.random.default_rng(2).random((40, 3)))
    torch.cuda.synchronize()
    assert rows > 5e5
    assert before - torch.cuda.mem_get_info()[0] < 97 * rows + 20 * 2**21
