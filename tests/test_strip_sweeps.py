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


@pytest.mark.parametrize('M_,N,K', [(128, 128, 32), (128, 128, 96), (256, 128, 224), (640, 640, 640), (640, 512, 288),
                                    (640, 768, 128), (1152, 1152, 128), (1152, 128, 1184)])
def test_tensor_core_product_over_shares(gpu_lib, M_, N, K):
    """The tensor-core product where a tile's K range is shared by one, two or four CTAs, evenly or not:
    against FP64, to the split scheme's bound (the existing comparison's 2e-5 of sum |a||b|)."""
    import ctypes as C
    import torch
    g = torch.Generator(device='cuda').manual_seed(M_ + 3 * N + 7 * K)
    A = torch.randn(M_, K, device='cuda', generator=g)
    B = torch.randn(N, K, device='cuda', generator=g)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)):
        C0 = torch.randn(M_, N, device='cuda', generator=g)
        out = C0.clone()
        st = gpu_lib.load().ocmp_dense_gemm_nt(1, M_, N, K, C.c_void_p(A.data_ptr()), K, C.c_void_p(B.data_ptr()), K,
                                               C.c_void_p(out.data_ptr()), N, alpha, beta,
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == gpu_lib.OK, gpu_lib.last_error()
        ref = alpha * (A.double() @ B.double().T) + beta * C0.double()
        scale = (A.double().abs() @ B.double().abs().T) + abs(beta) * C0.double().abs()
        assert ((out.double() - ref).abs() / scale).max().item() <= 2e-5
