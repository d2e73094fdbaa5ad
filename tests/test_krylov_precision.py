"""What the sums of the mixed-precision Krylov solves keep: systems whose FP32 products are all equal, so
that a long FP32 chain of them rounds the same way at every addition, and squares below FP32's normal
range."""
import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu

U = 2.0 ** -24      # unit roundoff of FP32


def _mass(n, batch=1, **kw):
    """P1 mass matrix of the unit square scaled to entries 12 and 2 (away from the boundary); its diagonal."""
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n)
    sp = fem.Space(m, 'H1', 1)
    A = fem.Matrix(sp, batch=batch, **kw)
    form = fem.make_form(mass=24.0 * n * n)
    A.assemble_batch([form] * batch) if batch > 1 else A.assemble(form)
    A1 = A
    if batch > 1:
        A1 = fem.Matrix(sp)
        A1.assemble(form)
    rp, col = sp.pattern()
    diag = np.flatnonzero(col == np.repeat(np.arange(sp.ndof), np.diff(rp)))
    return sp, A, A1, A1.device_values()[0][torch.as_tensor(diag, device='cuda')].clone()


def test_cg_curvature_is_summed_beyond_fp32(gpu_lib):
    """2,362,369 rows, about 60 per thread: one step from zero along z = D^-1 b, a constant c. x = alpha c
    with alpha = r.z / p.Ap; c, the row products and their products with c are made here in FP32 as the
    solve makes them. alpha and alpha c are rounded once each: 2 U, and as much for sums along the
    boundary. Summed in FP32 per thread, p.Ap is 10 U too large."""
    import torch
    from opencmp_gb300 import fem
    n = 1536
    sp, A, _, D = _mass(n, fp32=True)
    b = D.clone()
    x = torch.zeros_like(b)
    fem.KrylovSolver(A, method='CG', precision='mixed', tol=1e-12, maxit=1).solve(b, x, raise_on_fail=False)
    beta = float(torch.linalg.vector_norm(b))
    r = (b * (1.0 / beta)).float()
    z = (1.0 / D).float() * r
    f = np.float32
    inner = torch.isclose(D, torch.full_like(D, 12.0), rtol=1e-9)
    c = f(z[inner][0].item())
    assert int(inner.sum()) == (n - 1) ** 2 and bool((z[inner] == float(c)).all())
    # a row's seven products over four lanes: 2 + 2, 2 + 2, 2 + 2, 12; then two exchanges
    q = f(f(f(4) * c + f(4) * c) + f(f(4) * c + f(f(12) * c)))
    Az = torch.empty_like(b)
    A.mult(z.double(), Az)
    pap = float((z.double() * Az)[~inner].sum()) + float(c) * float(q) * int(inner.sum())
    alpha = float((r.double() * z.double()).sum()) / pap
    got = float(x[inner].mean()) / (beta * float(c))
    assert abs(got / alpha - 1) <= 4 * U, (got / alpha - 1) / U


def test_gmres_dots_are_summed_beyond_fp32(gpu_lib):
    """A batch of 262,144-row systems, a block each, so 256 rows per thread: one iteration from zero,
    x = D^-1 r (r.w) / (w.w) with w = A D^-1 r, at eighty scales of r = s D e. (e is 1/2 on a sixteenth of
    the rows: were w parallel to r, a second orthogonalisation would repair the sums.) Rounded in FP32:
    r (in w and in the dot product), D^-1, A D^-1, four additions of a row, w's scale twice, the products,
    y and x's two: 16 U in all. Summed in FP32 per thread, r.w is up to 60 U off."""
    import torch
    from opencmp_gb300 import fem
    B = 80
    sp, A, A1, D = _mass(511, batch=B, jacobi32=True)
    e = torch.ones_like(D)
    e[:sp.ndof // 16] = 0.5
    scales = 2.0 ** np.linspace(0, 1, B)
    b = torch.cat([s * D * e for s in scales])
    x = torch.zeros_like(b)
    fem.KrylovSolver(A, method='GMRES', restart=1, precision='mixed', tol=1e-12, maxit=1).solve_batch(
        b, x, raise_on_fail=False)
    w = torch.empty_like(D)
    A1.mult(e, w)                            # A D^-1 r = s A e
    c = float((D * e * w).sum() / (w * w).sum())
    err = [(float((x[q * sp.ndof:(q + 1) * sp.ndof] / (s * e)).mean()) / c - 1) / U for q, s in enumerate(scales)]
    assert max(map(abs, err)) <= 16, (min(err), max(err))


@pytest.mark.parametrize('scale', [1.0, 1e-31, 1e-33])
@pytest.mark.parametrize('path', ['csr', 'sell'])
def test_gmres_with_products_below_the_normal_range(gpu_lib, path, scale):
    """The last cycles' residuals are 1e-9 of the right-hand side's: their products with the basis are
    subnormal in FP32 but still add up."""
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(22)
    sp = fem.Space(m, 'H1', 1, m.bc_names)
    A = fem.Matrix(sp, jacobi32=True, dfloat=path == 'sell', sell=path == 'sell')
    A.assemble(fem.make_form(mass=1.0, diff=0.05, wind=(1.0, 0.5)))
    g = torch.Generator(device='cuda').manual_seed(3)
    b = scale * torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    sv = fem.KrylovSolver(A, method='GMRES', restart=30, precision='mixed', tol=1e-9, maxit=2000)
    info = sv.solve(b, torch.zeros_like(b), raise_on_fail=False)
    assert info.status == 0 and info.iterations <= 200, (info.status, info.iterations, info.relres)


@pytest.mark.parametrize('dim,n,order', [(2, 6, 1), (2, 24, 1), (2, 40, 2), (2, 100, 1), (3, 24, 1), (3, 56, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_cg_on_an_indefinite_matrix(gpu_lib, dim, n, order, precision):
    """-div grad - 30 (2D: one negative eigenvalue at 2 pi^2 - 30) or - 40 (3D: at 3 pi^2 - 40): CG goes on
    through steps of negative curvature. One block, all blocks' rows in shared memory, and streaming."""
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n) if dim == 2 else M.unit_cube(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, fp32=precision == 'mixed')
    A.assemble(fem.make_form(mass=-30.0 if dim == 2 else -40.0, diff=1.0))
    b = torch.zeros(sp.ndof, dtype=torch.float64, device='cuda')
    fem.assemble_rhs(sp, fem.make_form(diff=1.0), fem.make_rhs(src_const=1.0), b)
    info = fem.KrylovSolver(A, method='CG', precision=precision, tol=1e-9, maxit=2000).solve(b, torch.zeros_like(b),
                                                                                            raise_on_fail=False)
    assert info.status == 0 and info.relres <= 1e-9, (info.status, info.iterations, info.relres)


@pytest.mark.parametrize('n,most', [(16, 150), (24, 170), (32, 160)])
def test_pressure_solves_keep_what_they_reached(gpu_lib, n, most):
    """The Neumann pressure operator's constant mode is below FP32's rounding. An inner solve that steps along
    it as if it were negative curvature diverges, and the outer iteration pays: 450, 360 and 169 iterations
    when it did, 149, 164 and 156 when it stops there (and FP64: 149, 159, 156)."""
    import test_saddle as S
    th, A, b, u, sv = S._gpu_cavity(n, 'mixed', impl='host')
    info = sv.solve(b, u.clone(), raise_on_fail=False)
    assert info.status == 0 and info.iterations <= most, (info.status, info.iterations)
