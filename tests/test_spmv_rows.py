"""The operator application on either side of the sizes where its lanes per row change, against the same
product in torch. Both sum a row's products in FP64 in some order: 2 len eps sum |a||x| apart at most."""
import numpy as np
import pytest

from opencmp_gb300 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dim,kind,order,n', [(2, 'H1', 1, 5), (2, 'H1', 2, 20), (3, 'H1', 2, 26), (3, 'H1', 2, 27),
                                              (3, 'H1', 3, 13), (3, 'H1', 3, 15), (2, 'L2', 2, 113), (2, 'L2', 2, 115)])
def test_product_on_either_side_of_a_full_chip(gpu_lib, dim, kind, order, n):
    import torch
    from opencmp_gb300 import fem
    m = M.unit_square(n) if dim == 2 else M.unit_cube(n)
    sp = fem.Space(m, kind, order)
    A = fem.Matrix(sp)
    A.assemble(fem.make_form(mass=1.0, diff=0.05, wind=(1.0, 0.5, 0.25)[:dim], dg=kind == 'L2', ipc=10.0))
    x = torch.randn(sp.ndof, dtype=torch.float64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(n))
    y = torch.full_like(x, float('nan'))
    A.mult(x, y)
    rp, col = sp.pattern()
    row = torch.as_tensor(np.repeat(np.arange(sp.ndof), np.diff(rp)), device='cuda')
    t = A.device_values()[0] * x[torch.as_tensor(col, device='cuda').long()]
    ref = torch.zeros_like(x).index_add_(0, row, t)
    size = torch.zeros_like(x).index_add_(0, row, t.abs())
    assert bool(((y - ref).abs() <= 2 * int(np.diff(rp).max()) * 2.0 ** -52 * size).all())
