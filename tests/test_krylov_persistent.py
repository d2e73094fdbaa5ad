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
