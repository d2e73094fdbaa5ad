"""Batches and groups of more systems than SMs, each of few rows: several blocks per SM take them from a
queue. Every system against a dense solve, where the blocks' form changes (one free dof, the largest
system it takes and one above, a restart whose tables leave too few blocks, a partly filled last wave)
and for the operators' own data.

The bound is the residual's: |x - x*| / |x*| <= cond(A_ff) tol up to the data's own norm, so each system
is allowed 4 cond tol."""
import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _members(n, order, B, restart, precision, seed=0):
    import torch
    from opencmp_gb300 import fem
    mixed = precision == 'mixed'
    m = M.unit_square(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    rng = np.random.default_rng(seed + n)
    forms = [fem.make_form(mass=1.0, diff=float(10 ** rng.uniform(-2, -1)), wind=(1.0, float(rng.uniform(-1, 1))))
             for _ in range(B)]
    A = fem.Matrix(sp, batch=B, jacobi64=not mixed, jacobi32=mixed)
    A.assemble_batch(forms)
    b = torch.as_tensor(rng.standard_normal(B * sp.ndof), device='cuda')
    x0 = torch.as_tensor(rng.standard_normal(B * sp.ndof), device='cuda')
    sv = fem.KrylovSolver(A, method='GMRES', restart=restart, precision=precision, tol=TOL, maxit=3000)
    return sp, A, forms, b, x0, sv


def _check(sp, forms, b, x0, x, which):
    import torch
    from opencmp_gb300 import fem
    f = torch.as_tensor(sp.FreeDofs(), device='cuda')
    rp, col = sp.pattern()
    row = torch.as_tensor(np.repeat(np.arange(sp.ndof), np.diff(rp)), device='cuda')
    A1 = fem.Matrix(sp)
    for q in which:
        A1.assemble(forms[q])
        D = torch.zeros(sp.ndof, sp.ndof, dtype=torch.float64, device='cuda')
        D[row, torch.as_tensor(col, device='cuda').long()] = A1.device_values()[0]
        s = slice(q * sp.ndof, (q + 1) * sp.ndof)
        assert torch.equal(x[s][~f], x0[s][~f])
        if not bool(f.any()):
            continue
        rhs = (b[s] - D @ torch.where(f, torch.zeros_like(x0[s]), x0[s]))[f]
        Aff = D[f][:, f]
        ref = torch.linalg.solve(Aff, rhs)
        bound = 4 * float(torch.linalg.cond(Aff)) * TOL * max(float(ref.norm()), float(rhs.norm()))
        assert float((x[s][f] - ref).norm()) <= bound, q


@pytest.mark.parametrize('n,order,B,restart', [(2, 1, 5000, 30), (1, 1, 200, 5), (4, 2, 153, 30), (9, 2, 700, 7),
                                               (31, 1, 160, 30), (32, 1, 160, 30), (8, 2, 300, 100), (5, 3, 2000, 20)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_many_small_systems(gpu_lib, n, order, B, restart, precision):
    import torch
    sp, A, forms, b, x0, sv = _members(n, order, B, restart, precision)
    xs = []
    for _ in range(2):
        x = x0.clone()
        infos = sv.solve_batch(b, x)
        assert all(i.status == 0 and i.relres <= TOL for i in infos)
        xs.append(x)
    assert torch.equal(*xs)
    _check(sp, forms, b, x0, xs[0], {0, B // 2, B - 1})


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_group_of_many_small_systems(gpu_lib, precision):
    import torch
    from opencmp_gb300 import fem
    parts = [_members(n, order, B, 25, precision, seed=3) for n, order, B in ((3, 1, 90), (7, 2, 60), (6, 3, 50))]
    group = fem.KrylovGroup([p[-1] for p in parts])
    xs = [p[4].clone() for p in parts]
    infos = group.solve([p[3] for p in parts], xs)
    assert len(infos) == 200 and all(i.status == 0 and i.relres <= TOL for i in infos)
    for (sp, A, forms, b, x0, sv), x in zip(parts, xs):
        _check(sp, forms, b, x0, x, {0, len(forms) - 1})


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_large_systems_in_a_large_group(gpu_lib, precision):
    """Systems whose share of the blocks would be small for their rows go one after another through teams of
    blocks, the smaller ones one per block afterwards: each meets its tolerance, by the matrix too, and
    equals its own solve to it (mass-dominated: condition below 1e4)."""
    import torch
    from opencmp_gb300 import fem
    parts = [_members(n, order, B, 20, precision, seed=5) for n, order, B in ((128, 2, 40), (32, 2, 30), (4, 1, 50))]
    group = fem.KrylovGroup([p[-1] for p in parts])
    runs = []
    for _ in range(2):
        xs = [p[4].clone() for p in parts]
        infos = group.solve([p[3] for p in parts], xs)
        assert len(infos) == 120 and all(i.status == 0 and i.relres <= TOL for i in infos)
        runs.append(xs)
    assert all(torch.equal(u, v) for u, v in zip(*runs))
    mixed = precision == 'mixed'
    for (sp, A, forms, b, x0, sv), x in zip(parts, runs[0]):
        f = torch.as_tensor(sp.FreeDofs(), device='cuda')
        A1 = fem.Matrix(sp, jacobi64=not mixed, jacobi32=mixed)
        for q in {0, len(forms) // 2, len(forms) - 1}:
            A1.assemble(forms[q])
            s = slice(q * sp.ndof, (q + 1) * sp.ndof)
            y = x0[s].clone()
            fem.KrylovSolver(A1, method='GMRES', restart=20, precision=precision, tol=TOL, maxit=3000).solve(
                b[s].contiguous(), y)
            assert torch.equal(x[s][~f], y[~f])
            assert float((x[s] - y).norm()) <= 2 * 1e4 * TOL * max(float(y.norm()), float(b[s].norm()))
