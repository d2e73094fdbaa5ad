"""Krylov handles after a solve that failed: the next solve equals a fresh handle's bit for bit.

A mixed-precision GMRES handle after a solve that ended non-finite. The right-hand side is finite in FP64 but above FP32's range, so the basis holds
infinities from its first vector on; the sizes are FP32 systems of 512 or more rows a block (tiles of
128 rows, 16-byte loads) whose last tile is not full.

Any handle after a wait of one block for another that ran out (the blocks are made to wait for an
arrival, or a word, that does not come; the wait's limit is half a millisecond then): OCMP_TIMEOUT."""
import ctypes as C

import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _system(n, order, batch=1, sell=False):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, batch=batch, jacobi32=True, dfloat=sell, sell=sell)
    forms = [fem.make_form(mass=1.0, diff=0.05 + 0.01 * q, wind=(1.0, 0.5)) for q in range(batch)]
    A.assemble_batch(forms) if batch > 1 else A.assemble(forms[0])
    g = torch.Generator(device='cuda').manual_seed(n)
    b = torch.randn(batch * sp.ndof, dtype=torch.float64, device='cuda', generator=g)
    return sp, A, b


def _solver(A, precond='jacobi'):
    from opencmp_gb300 import fem
    sv = fem.KrylovSolver(A, method='GMRES', restart=20, precond=precond, precision='mixed', tol=1e-10, maxit=20000)
    sv.update()
    return sv


@pytest.mark.parametrize('n,order,path', [(22, 1, 'csr'), (30, 1, 'sell'), (15, 2, 'csr'), (22, 1, 'strip'), (30, 1, 'strip'),
                                          (141, 2, 'sell')])
def test_solve_after_a_non_finite_one(gpu_lib, n, order, path):
    import torch
    from opencmp_gb300 import _lib as LB
    sp, A, b = _system(n, order, sell=path == 'sell')
    assert sp.ndof % 128 != 0 and sp.ndof >= 512
    pre = 'strip' if path == 'strip' else 'jacobi'
    sv = _solver(A, pre)
    bad = sv.solve(1e39 * b, torch.zeros_like(b), raise_on_fail=False)
    assert bad.status == LB.ERR_NONFINITE
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    info, ref = sv.solve(b, x, raise_on_fail=False), _solver(A, pre).solve(b, y)
    assert info.status == 0 and info.iterations == ref.iterations
    assert torch.equal(x, y)


def test_batch_and_group_after_a_non_finite_solve(gpu_lib):
    import torch
    from opencmp_gb300 import _lib as LB, fem
    sp, A, b = _system(22, 1, batch=3)
    sv = _solver(A)
    bad = sv.solve_batch(1e39 * b, torch.zeros_like(b), raise_on_fail=False)
    assert all(i.status == LB.ERR_NONFINITE for i in bad)
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    assert all(i.status == 0 for i in sv.solve_batch(b, x, raise_on_fail=False))
    _solver(A).solve_batch(b, y)
    assert torch.equal(x, y)
    sp2, A2, b2 = _system(30, 1)
    members = [_solver(A), _solver(A2)]
    group = fem.KrylovGroup(members)
    big = [1e39 * b, 1e39 * b2]
    assert all(i.status == LB.ERR_NONFINITE for i in group.solve(big, [torch.zeros_like(v) for v in big],
                                                                 raise_on_fail=False))
    xs = [torch.zeros_like(b), torch.zeros_like(b2)]
    assert all(i.status == 0 for i in group.solve([b, b2], xs, raise_on_fail=False))
    ys = [torch.zeros_like(b), torch.zeros_like(b2)]
    fem.KrylovGroup([_solver(A), _solver(A2)]).solve([b, b2], ys)
    assert all(torch.equal(u, v) for u, v in zip(xs, ys))


@pytest.mark.parametrize('method,precond,n,order,which', [('CG', 'jacobi', 40, 2, 0), ('CG', 'jacobi', 500, 1, 0),
                                                          ('GMRES', 'jacobi', 40, 2, 0), ('GMRES', 'strip', 60, 1, 0),
                                                          ('GMRES', 'strip', 60, 1, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_solve_after_a_wait_that_ran_out(gpu_lib, method, precond, n, order, which, precision):
    import torch
    from opencmp_gb300 import _lib as LB, fem
    m = M.unit_square(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, fp32=precision == 'mixed')
    A.assemble(fem.make_form(mass=1.0, diff=0.05))
    b = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(n))

    def solver():
        sv = fem.KrylovSolver(A, method=method, restart=20, precond=precond, precision=precision, tol=1e-9, maxit=3000)
        sv.update()
        return sv

    starve = LB.load().ocmp_test_starve
    starve.argtypes, starve.restype = [C.c_void_p, C.c_int32], C.c_int
    y = torch.zeros_like(b)
    ref = solver().solve(b, y)
    sv = solver()
    for _ in range(2):
        assert starve(sv.h, which) == 0
        with pytest.raises(LB.OcmpError) as e:
            sv.solve(b, torch.zeros_like(b))
        assert e.value.status == LB.TIMEOUT
        for _ in range(2):
            x = torch.zeros_like(b)
            info = sv.solve(b, x)
            assert info.iterations == ref.iterations and torch.equal(x, y)


@pytest.mark.parametrize('n,order,batch', [(40, 1, 20), (128, 2, 40)])
def test_batch_after_a_wait_that_ran_out(gpu_lib, n, order, batch):
    """Twenty teams of seven blocks; teams of four that take systems of 66,049 rows from a queue."""
    import torch
    from opencmp_gb300 import _lib as LB
    sp, A, b = _system(n, order, batch=batch)
    y = torch.zeros_like(b)
    _solver(A).solve_batch(b, y)
    sv = _solver(A)
    starve = LB.load().ocmp_test_starve
    starve.argtypes, starve.restype = [C.c_void_p, C.c_int32], C.c_int
    assert starve(sv.h, 0) == 0
    with pytest.raises(LB.OcmpError) as e:
        sv.solve_batch(b, torch.zeros_like(b))
    assert e.value.status == LB.TIMEOUT
    x = torch.zeros_like(b)
    sv.solve_batch(b, x)
    assert torch.equal(x, y)
