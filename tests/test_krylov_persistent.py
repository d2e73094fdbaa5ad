"""The persistent Krylov kernels (a whole solve in one cooperative launch) at the sizes where their
split over blocks changes: no free dof, one block, the first size of two, a ragged last tile, one
block per SM with many tiles each; against a dense FP64 solve of the same matrix.

The error bound is the residual's: |x - x*| / |x*| <= cond(A_ff) tol up to the data's own norm, so
each case allows 4 cond tol (the solve is asked for tol in the norm of the right-hand side)."""
import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _dense(sp, A):
    rp, col = sp.pattern()
    D = np.zeros((sp.ndof, sp.ndof))
    D[np.repeat(np.arange(sp.ndof), np.diff(rp)), col] = A.values()
    return D


def _reference(sp, A, b, x0):
    import torch
    D = torch.as_tensor(_dense(sp, A), device='cuda')
    f = torch.as_tensor(sp.FreeDofs(), device='cuda')
    x = x0.clone()
    if not bool(f.any()):
        return x, 1.0
    Aff = D[f][:, f]
    x[f] = torch.linalg.solve(Aff, (b - D @ torch.where(f, torch.zeros_like(x), x))[f])
    return x, float(torch.linalg.cond(Aff))


def _problem(dim, n, order, mixed=False, seed=0):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n) if dim == 2 else M.unit_cube(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, fp32=mixed)
    form = fem.make_form(mass=1.0, diff=0.05)
    A.assemble(form)
    g = torch.Generator(device='cuda').manual_seed(seed + 31 * n + order)
    b = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    x0 = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)   # Dirichlet values and guess
    return sp, A, b, x0


@pytest.mark.parametrize('dim,n,order', [(2, 1, 1), (2, 2, 1), (2, 21, 1), (2, 22, 1), (2, 8, 3), (2, 24, 2), (3, 5, 2),
                                         (3, 3, 3), (2, 33, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_cg_in_one_launch(gpu_lib, dim, n, order, precision):
    from opencmp_gb300 import fem
    import torch
    tol = 1e-12
    sp, A, b, x0 = _problem(dim, n, order, precision == 'mixed')
    ref, cond = _reference(sp, A, b, x0)
    sv = fem.KrylovSolver(A, method='CG', precision=precision, tol=tol, maxit=2000)
    xs = []
    for _ in range(2):
        x = x0.clone()
        info = sv.solve(b, x)
        assert info.status == 0 and info.relres <= tol
        xs.append(x)
    assert torch.equal(xs[0], xs[1])                        # the sums have a fixed order
    f = torch.as_tensor(sp.FreeDofs(), device='cuda')
    assert torch.equal(xs[0][~f], x0[~f])
    scale = float(torch.linalg.vector_norm(ref)) + 1e-300
    assert float(torch.linalg.vector_norm(xs[0] - ref)) <= 4 * cond * tol * max(scale, float(torch.linalg.vector_norm(b)))


@pytest.mark.parametrize('n', [2, 40])
def test_cg_stops_and_reports(gpu_lib, n):
    """The iteration cap, a non-finite right-hand side and a converged start, on one block and on
    several; the solver stays usable after each."""
    from opencmp_gb300 import _lib as LB, fem
    sp, A, b, x0 = _problem(2, n, 2)
    sv = fem.KrylovSolver(A, method='CG', tol=1e-12, maxit=2)
    info = sv.solve(b, x0.clone(), raise_on_fail=False)
    assert info.status == LB.NOT_CONVERGED and info.iterations == 2 and 0 < info.relres
    bad = b.clone()
    bad[int(np.flatnonzero(sp.FreeDofs())[0])] = float('nan')
    assert sv.solve(bad, x0.clone(), raise_on_fail=False).status == LB.ERR_NONFINITE
    sv = fem.KrylovSolver(A, method='CG', tol=1e-12, maxit=2000)
    x = x0.clone()
    assert sv.solve(b, x).status == 0
    # the solution's own residual may sit a rounding above the tolerance it was stopped at
    sv2 = fem.KrylovSolver(A, method='CG', tol=1e-11, maxit=2000)
    y = x.clone()
    info = sv2.solve(b, y)
    assert info.iterations == 0 and info.relres0 <= 1e-11 and bool((x == y).all())


def _convection(dim, n, order, mixed, sell=False):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n) if dim == 2 else M.unit_cube(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, jacobi32=mixed, jacobi64=not mixed, dfloat=sell, sell=sell)
    A.assemble(fem.make_form(mass=1.0, diff=0.05, wind=(1.0, 0.5, 0.25)[:dim]))
    g = torch.Generator(device='cuda').manual_seed(7 * n + order)
    b = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    x0 = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    return sp, A, b, x0


# one free dof's worth of rows, one block, the first sizes of two blocks in FP64 and FP32, ragged last
# tiles, tiles of 128 rows (FP32, 512 rows a block), a restart shorter than the solve, the largest restart
@pytest.mark.parametrize('dim,n,order,restart', [(2, 1, 1, 5), (2, 2, 1, 5), (2, 21, 1, 30), (2, 22, 1, 7), (2, 31, 1, 30),
                                                 (2, 24, 2, 30), (2, 12, 3, 128), (3, 5, 2, 30), (3, 3, 3, 40)])
@pytest.mark.parametrize('path', ['fp64', 'mixed', 'sell'])
def test_gmres_in_one_launch(gpu_lib, dim, n, order, restart, path):
    from opencmp_gb300 import fem
    import torch
    tol = 1e-11
    sp, A, b, x0 = _convection(dim, n, order, path != 'fp64', path == 'sell')
    ref, cond = _reference(sp, A, b, x0)
    sv = fem.KrylovSolver(A, method='GMRES', restart=restart, precision='fp64' if path == 'fp64' else 'mixed', tol=tol,
                          maxit=5000)
    xs = []
    for _ in range(2):
        x = x0.clone()
        info = sv.solve(b, x)
        assert info.status == 0 and info.relres <= tol
        xs.append(x)
    assert torch.equal(xs[0], xs[1])
    f = torch.as_tensor(sp.FreeDofs(), device='cuda')
    assert torch.equal(xs[0][~f], x0[~f])
    scale = max(float(torch.linalg.vector_norm(ref)), float(torch.linalg.vector_norm(b)), 1e-300)
    assert float(torch.linalg.vector_norm(xs[0] - ref)) <= 4 * cond * tol * scale


def test_gmres_tiles_of_128_rows(gpu_lib):
    """FP32 systems of 512 rows a block on every SM read their basis 16 bytes at a time: the iteration
    and the solution agree with the FP64 solve of the same system to the tolerance asked for."""
    import torch
    from opencmp_gb300 import fem
    tol = 1e-11
    out = {}
    for path in ('fp64', 'sell'):
        sp, A, b, x0 = _convection(2, 141, 2, path != 'fp64', path == 'sell')      # 80,089 dofs
        x = x0.clone()
        info = fem.KrylovSolver(A, method='GMRES', restart=20, precision='fp64' if path == 'fp64' else 'mixed', tol=tol,
                                maxit=3000).solve(b, x)
        assert info.status == 0 and info.relres <= tol
        out[path] = x
    # both residuals are below tol |b|; the matrices are mass-dominated (condition below 1e4)
    d = float(torch.linalg.vector_norm(out['fp64'] - out['sell']) / torch.linalg.vector_norm(out['fp64']))
    assert d <= 2 * 1e4 * tol


@pytest.mark.parametrize('order,n', [(1, 3), (2, 5), (2, 17), (3, 9)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_gmres_block_jacobi_in_one_launch(gpu_lib, order, n, precision):
    """Element blocks of 3, 6 and 10 rows stay whole in their tiles; against a dense solve."""
    import torch
    from opencmp_gb300 import fem
    tol = 1e-11
    m = M.unit_square(n)
    sp = fem.Space(m, 'L2', order)
    A = fem.Matrix(sp)
    A.assemble(fem.make_form(mass=1.0, diff=0.01, dt=0.1, wind=(1.0, 0.5), dg=True, ipc=10.0,
                             nitsche_mask=m.label_mask(m.bc_names)))
    g = torch.Generator(device='cuda').manual_seed(n)
    b = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    x = torch.zeros_like(b)
    info = fem.KrylovSolver(A, method='GMRES', restart=30, precond='block_jacobi', precision=precision, tol=tol,
                            maxit=3000).solve(b, x)
    assert info.status == 0 and info.relres <= tol
    ref, cond = _reference(sp, A, b, torch.zeros_like(b))
    scale = max(float(torch.linalg.vector_norm(ref)), float(torch.linalg.vector_norm(b)))
    assert float(torch.linalg.vector_norm(x - ref)) <= 4 * cond * tol * scale


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_group_of_very_uneven_systems(gpu_lib, precision):
    """Teams of several blocks, single blocks of the queue, and more systems than blocks: every system
    meets its tolerance and equals its own solve to it."""
    import torch
    from opencmp_gb300 import fem
    tol = 1e-10
    mixed = precision == 'mixed'
    members, bs, xs, refs = [], [], [], []
    for n, order, B in ((2, 1, 90), (6, 2, 80), (40, 2, 2), (9, 3, 7)):
        m = M.unit_square(n)
        sp = fem.Space(m, 'H1', order, m.bc_names)
        forms = [fem.make_form(mass=0.1, diff=0.02 + 0.01 * q, wind=(1.0, 0.3)) for q in range(B)]
        A = fem.Matrix(sp, batch=B, jacobi32=mixed, jacobi64=not mixed)
        A.assemble_batch(forms)
        g = torch.Generator(device='cuda').manual_seed(n)
        b = torch.randn(B * sp.ndof, dtype=torch.float64, device='cuda', generator=g)
        members.append(fem.KrylovSolver(A, method='GMRES', restart=25, precision=precision, tol=tol, maxit=3000))
        bs.append(b)
        xs.append(torch.zeros_like(b))
        A1 = fem.Matrix(sp, jacobi32=mixed, jacobi64=not mixed)
        A1.assemble(forms[B - 1])
        x1 = torch.zeros(sp.ndof, dtype=torch.float64, device='cuda')
        fem.KrylovSolver(A1, method='GMRES', restart=25, precision=precision, tol=tol, maxit=3000).solve(
            b[(B - 1) * sp.ndof:].clone(), x1)
        refs.append(x1)
    group = fem.KrylovGroup(members)
    for _ in range(2):
        for x in xs:
            x.zero_()
        infos = group.solve(bs, xs)
        assert all(i.status == 0 and i.relres <= tol for i in infos) and len(infos) == 179
    for x, r in zip(xs, refs):
        d = float(torch.linalg.vector_norm(x[-r.numel():] - r) / torch.linalg.vector_norm(r))
        assert d <= 2 * 1e4 * tol
