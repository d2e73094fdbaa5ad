"""Krylov handles and their neighbours used from several host threads, a handle each; what a handle of many
tiny systems holds; the products that a handle counts."""
import ctypes as C
import threading

import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _system(n, order, **kw):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n)
    sp = fem.Space(m, 'H1', order, m.bc_names)
    A = fem.Matrix(sp, **kw)
    A.assemble(fem.make_form(mass=1.0, diff=0.05))
    b = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(n))
    return sp, A, b


def _side_by_side(jobs, rounds=20000):
    """jobs: (entry point, arguments but the stream, index of the stream argument, results). Each in a
    thread and on a stream of its own, over and over: every call succeeds, and the results at the end
    are those of the calls made alone."""
    import torch
    from opencmp_gb300 import _lib as LB
    streams = [torch.cuda.Stream() for _ in jobs]
    calls = []
    for (fn, args, at, out), st in zip(jobs, streams):
        args = list(args)
        args.insert(at, C.c_void_p(st.cuda_stream))
        assert fn(*args) == 0, LB.last_error()
        torch.cuda.synchronize()
        calls.append((fn, args, out, [t.clone() for t in out]))
    errors, start = [], threading.Barrier(len(jobs))

    def work(fn, args):
        start.wait()
        for _ in range(rounds):
            if fn(*args):
                errors.append(LB.last_error())
                return

    ts = [threading.Thread(target=work, args=c[:2]) for c in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for _, _, out, ref in calls:
        assert all(torch.equal(u, v) for u, v in zip(out, ref))


def _ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize('method,small,large', [('CG', (2, 1, 5), (64, 2, 5)), ('GMRES', (2, 1, 5), (2, 1, 120))])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_threads_with_a_solver_each(gpu_lib, method, small, large, precision):
    """Solvers whose launches take little and much shared memory (matrix rows a block; restart), from
    solutions that need no further step."""
    import torch
    from opencmp_gb300 import _lib as LB, fem
    jobs, keep = [], []
    for n, order, restart in (small, large, small, large):
        sp, A, b = _system(n, order, fp32=precision == 'mixed')
        x = torch.zeros_like(b)
        kw = dict(method=method, restart=restart, precision=precision, maxit=2000)
        fem.KrylovSolver(A, tol=1e-10, **kw).solve(b, x)
        sv, info = fem.KrylovSolver(A, tol=1e-8, **kw), LB.SolveInfo()
        keep.append((sv, b, info))
        jobs.append((LB.load().ocmp_solve, (sv.h, _ptr(b), _ptr(x), C.byref(info)), 3, [x]))
    torch.cuda.synchronize()
    _side_by_side(jobs)


def test_threads_with_a_network_each(gpu_lib):
    """Networks of one and eight features."""
    import torch
    from opencmp_gb300 import _lib as LB
    from opencmp_gb300.guess import GuessNet
    jobs, keep = [], []
    for F in (1, 8, 1, 8):
        net, loss = GuessNet(F, seed=F), C.c_double(0)
        g = torch.Generator(device='cuda').manual_seed(F)
        X = torch.randn(300, F, device='cuda', generator=g)
        T = torch.randn(300, device='cuda', generator=g)
        grad = np.zeros(net.nparams, np.float32)
        keep.append((net, X, T, loss, grad))
        jobs.append((LB.load().ocmp_guess_loss_grad,
                     (net.h, _ptr(X), _ptr(T), C.c_int64(300), C.byref(loss), C.c_void_p(grad.ctypes.data)), 6,
                     [torch.from_numpy(grad)]))
    torch.cuda.synchronize()
    _side_by_side(jobs)


def test_threads_with_a_matrix_each(gpu_lib):
    """Assemblies with facet terms stage their longest row in shared memory: 7 entries on a square's
    vertices, 151 at the centre of a polygon."""
    import torch
    from opencmp_gb300 import _lib as LB, fem
    k = 150
    ang = 2 * np.pi * np.arange(k) / k
    ring = np.stack([np.arange(1, k + 1), np.roll(np.arange(1, k + 1), -1)], 1).astype(np.int32)
    fan = M.Mesh(np.concatenate([np.zeros((1, 2)), np.stack([np.cos(ang), np.sin(ang)], 1)]),
                 np.concatenate([np.zeros((k, 1), np.int32), ring], 1), ring, np.zeros(k, np.int32), ['rim'])
    jobs, keep = [], []
    for m in (M.unit_square(8), fan, M.unit_square(8), fan):
        sp = fem.Space(m, 'H1', 1)
        A, form = fem.Matrix(sp), fem.make_form(mass=1.0, diff=0.1, robin={0: 0.5})
        keep.append((A, form))
        jobs.append((LB.load().ocmp_assemble_matrix, (A.h, C.byref(form)), 2, [A.device_values()[0]]))
    torch.cuda.synchronize()
    _side_by_side(jobs)


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_memory_of_a_batch_of_tiny_systems(gpu_lib, precision):
    """The bases of 9-dof systems take (restart + 1) vectors of at most 16 values each."""
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(2)
    sp = fem.Space(m, 'H1', 1, m.bc_names)
    B, restart = 20000, 30
    A = fem.Matrix(sp, batch=B, jacobi64=precision == 'fp64', jacobi32=precision == 'mixed')
    small = 8 * (restart * (restart + 1) // 2 + 4 * restart + 8) * B        # Hessenberg matrices, rotations
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    sv = fem.KrylovSolver(A, method='GMRES', restart=restart, precision=precision, tol=1e-8, maxit=10)
    torch.cuda.synchronize()
    used = free0 - torch.cuda.mem_get_info()[0]
    basis = (8 if precision == 'fp64' else 4) * (restart + 1) * 16 * B
    # beside these a few vectors and results per system, and the allocator's granularity
    assert used <= small + basis + 1000 * B + (64 << 20), (used, small, basis)
    assert sv.h


@pytest.mark.parametrize('precond', ['jacobi', 'strip'])
@pytest.mark.parametrize('n', [2, 12, 60])
def test_every_product_is_counted(gpu_lib, precond, n):
    import torch
    from opencmp_gb300 import fem
    sp, A, b = _system(n, 1)
    sv = fem.KrylovSolver(A, method='GMRES', restart=30, precond=precond, tol=1e-10, maxit=2000)
    sv.update()
    sv.spmv_timing(True)
    total = 0
    for _ in range(3):
        total += sv.solve(b, torch.zeros_like(b)).iterations
        # one more may be queued past convergence with the strip; it does no product
        count, ms = sv.spmv_stats()
        assert count == total and ms >= 0.0


def test_graph_switch_is_accepted_for_gmres_and_changes_nothing(gpu_lib):
    import torch
    from opencmp_gb300 import _lib as LB, fem
    sp, A, b = _system(20, 2)
    xs = []
    for on in (False, True):
        sv = fem.KrylovSolver(A, method='GMRES', restart=20, tol=1e-10, maxit=500)
        sv.set_graph(on)
        xs.append(torch.zeros_like(b))
        sv.solve(b, xs[-1])
    assert torch.equal(*xs)
    for kw in (dict(method='CG'), dict(method='GMRES', precond='strip')):
        with pytest.raises(LB.OcmpError) as e:
            fem.KrylovSolver(A, tol=1e-10, **kw).set_graph(True)
        assert e.value.status == LB.ERR_UNSUPPORTED
