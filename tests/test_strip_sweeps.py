"""The strip preconditioner's two sweeps (one cooperative launch) at the sizes where its steps change:
one strip, two, an odd and an even number, strips whose rows do not fit in shared memory, coupling
lists longer and shorter than the blocks' threads, constrained dofs, both vector types, and in place
(GMRES applies it to its own correction).

GMRES is asked for tol and stops on its true residual, so the residual recomputed here from the matrix
in FP64 may exceed tol by its own rounding only: 64 eps |A| |x| / |b| stays below tol / 100 at these sizes. An exact inverse
in FP32 reaches 1e-10 within a few iterations; twenty allow for condition numbers up to 1e6."""
import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize('dim,kind,order,n', [(2, 'H1', 1, 3), (2, 'L2', 1, 5), (2, 'H1', 1, 40), (2, 'H1', 1, 90),
                                              (2, 'L2', 2, 24), (2, 'L2', 3, 20), (2, 'L2', 1, 70), (2, 'H1', 2, 24),
                                              (3, 'H1', 1, 16), (3, 'H1', 2, 7)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_sweeps_in_one_launch(gpu_lib, dim, kind, order, n, precision):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n) if dim == 2 else M.unit_cube(n)
    dg = kind == 'L2'
    sp = fem.Space(m, kind, order, () if dg else m.bc_names)
    rng = np.random.default_rng(n + 10 * order)
    W = torch.as_tensor(rng.standard_normal((m.nv, dim)), device='cuda')
    form = fem.make_form(diff=0.05, mass=1.0, wind_vtx=W, dg=dg, ipc=10.0,
                         nitsche_mask=m.label_mask(m.bc_names) if dg else 0)
    A = fem.Matrix(sp, fp32=precision == 'mixed')
    A.assemble(form)
    b = torch.as_tensor(rng.standard_normal(sp.ndof), device='cuda')
    x0 = torch.as_tensor(rng.standard_normal(sp.ndof), device='cuda')
    sv = fem.KrylovSolver(A, method='GMRES', restart=20, precond='strip', precision=precision, tol=TOL, maxit=60)
    sv.update()
    rp, col = sp.pattern()
    S = torch.sparse_csr_tensor(torch.as_tensor(rp), torch.as_tensor(col.astype(np.int64)), torch.as_tensor(A.values()),
                                (sp.ndof, sp.ndof)).cuda()
    free = torch.as_tensor(sp.FreeDofs(), device='cuda').bool()
    r0 = (b - S @ torch.where(free, torch.zeros_like(x0), x0))[free].norm().item()
    xs = []
    for _ in range(2):
        x = x0.clone()
        info = sv.solve(b, x)
        assert info.status == 0 and info.iterations <= 20, (info.status, info.iterations, info.relres)
        xs.append(x)
    assert torch.equal(xs[0], xs[1])
    r = (b - S @ xs[0])[free].norm().item()
    assert r <= TOL * 1.01 * r0, (r, r0, info.iterations)
    assert torch.equal(xs[0][~free], x0[~free])
