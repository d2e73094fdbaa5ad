"""What the sums of the mixed-precision Krylov solves keep: systems whose FP32 products are all equal, so
that a long FP32 chain of them rounds the same way at every addition."""
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
