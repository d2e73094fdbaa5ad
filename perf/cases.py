"""The work a user of this framework has it do, as measurable cases.

Every family is one unit of work of a simulation, through the package's public objects (``fem``,
``saddle``, ``guess``), at the sizes the test fixtures, the configurations of ``bench.py`` and the
drop-in runs use:

  elliptic   a diffusion solve with Jacobi-CG: assemble, load vector, preconditioner update, solve;
             stationary (Poisson, ``dt`` 0) or one implicit-Euler step of the heat equation
  transport  one implicit-Euler step of convection-diffusion on a continuous space: assemble, mass
             load, update, GMRES + Jacobi (``path`` 'fp64': the default of a run; 'mixed':
             double-float assembly, FP32 inner iteration on the SELL-32 copy, FP64 refinement)
  dg         one implicit-Euler step of convection-diffusion on a discontinuous space (facet terms,
             block-Jacobi GMRES)
  direct     a DG convection-diffusion step solved with the strip factorisation, refactorised on every
             call as a direct linear solver does
  ins        one Euler-IMEX step of the lid-driven cavity on Taylor-Hood elements
  batch      many uneven steady instances assembled and solved by one solver group
  apply      an operator application y = A x, what an explicit time step or a user's own loop calls
  train      one training evaluation of the learned initial guess: forward, residual loss, backward

A run solves to the 1e-12 relative residual the drop-in uses for OpenCMP's default linear solver, at
sizes where 64-bit residuals get there (the transport steps of order 3 to 1e-13: their hierarchical
basis turns a residual into a thousand times the error), so the solutions do not depend on where an
iteration happens to stop.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from opencmp_gb300 import _lib as LB
from opencmp_gb300 import fem
from opencmp_gb300 import mesh as M

TOL = 1e-12
TOL_P3 = 1e-13


def listed():
    return [
        # a coarse test-fixture run: every call is latency
        dict(name='elliptic_2d_p2_n8', family='elliptic', dim=2, order=2, n=8, path='fp64', dt=0.0),
        # the Poisson configuration of the benchmark set: 64 x 64 x 2, P2
        dict(name='elliptic_2d_p2_n64', family='elliptic', dim=2, order=2, n=64, path='fp64', dt=0.0),
        # linear tetrahedra with the mixed-precision option
        dict(name='elliptic_3d_p1_n44_mixed', family='elliptic', dim=3, order=1, n=44, path='mixed', dt=0.0),
        # a small transient run, an odd mesh
        dict(name='transport_2d_p1_n33', family='transport', dim=2, order=1, n=33, path='fp64', wind='const'),
        # an ordinary 3D run with a space-dependent wind, FP64 throughout
        dict(name='transport_3d_p2_n21_vertex', family='transport', dim=3, order=2, n=21, path='fp64', wind='vertex'),
        # the benchmark's mesh (64^3 x 6 tetrahedra, P2) on the mixed path: the largest
        dict(name='transport_3d_p2_n64_mixed', family='transport', dim=3, order=2, n=64, path='mixed', wind='const'),
        # a transient discontinuous Galerkin run
        dict(name='dg_2d_p2_n72', family='dg', order=2, n=72),
        # the direct solve of a discontinuous Galerkin system, tensor-core products
        dict(name='direct_dg_p2_n96', family='direct', order=2, n=96, gemm='tensor'),
        # a Navier-Stokes step at half the benchmark's mesh
        dict(name='ins_p2_n128', family='ins', order=2, n=128, path='fp64'),
        # many small problems at once
        dict(name='batch_48', family='batch', count=48, nmax=48, restart=50),
        # one operator application, quadratic tetrahedra
        dict(name='apply_3d_p2_n40', family='apply', dim=3, order=2, n=40),
        # training the initial guess on a mid-size transient run
        dict(name='train_3d_p2_n28', family='train', dim=3, order=2, n=28, history=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# the largest mesh of each (dimension, order) drawn
_NMAX = {(2, 1): 256, (2, 2): 160, (2, 3): 110, (3, 1): 60, (3, 2): 48, (3, 3): 24}
# and of a stationary solve, whose 64-bit residual floor grows like the square of the mesh
_NMAX_POISSON = {(2, 1): 96, (2, 2): 64, (2, 3): 24, (3, 1): 44, (3, 2): 20, (3, 3): 8}


def draw(rng):
    family = rng.choice(['elliptic', 'elliptic', 'transport', 'transport', 'transport', 'dg', 'direct', 'ins', 'batch',
                         'apply', 'train'])
    if family in ('elliptic', 'transport', 'apply', 'train'):
        dim = rng.choice([2, 3])
        order = rng.choice([1, 2, 3])
        dt = rng.choice([0.0, 1e-3]) if family == 'elliptic' else 1e-3
        n = _log_int(rng, 6 if dim == 2 else 4, (_NMAX if dt else _NMAX_POISSON)[(dim, order)])
        c = dict(family=family, dim=dim, order=order, n=n)
        if family == 'elliptic':
            c.update(path=rng.choice(['fp64', 'fp64', 'mixed']) if order < 3 else 'fp64', dt=dt)
        elif family == 'transport':
            c.update(path=rng.choice(['fp64', 'mixed']) if order < 3 else 'fp64', wind=rng.choice(['const', 'vertex']))
        elif family == 'train':
            c['history'] = rng.choice([4, 5, 6])
        return c
    if family == 'dg':
        order = rng.choice([1, 2, 3])
        return dict(family='dg', order=order, n=_log_int(rng, 6, {1: 160, 2: 110, 3: 70}[order]))
    if family == 'direct':
        order = rng.choice([1, 2])
        return dict(family='direct', order=order, n=_log_int(rng, 12, {1: 150, 2: 100}[order]),
                    gemm=rng.choice(['simt', 'tensor']))
    if family == 'ins':
        return dict(family='ins', order=2, n=_log_int(rng, 10, 150), path=rng.choice(['fp64', 'mixed']))
    return dict(family='batch', count=_log_int(rng, 4, 56), nmax=_log_int(rng, 12, 48), restart=rng.choice([30, 50]))


# ---------------------------------------------------------------- inputs
def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float64), device='cuda')


def _field(rng, dim, modes=4):
    """A smooth random field on the unit square or cube: a few plane waves."""
    k = rng.integers(1, 4, (modes, dim)) * math.pi
    a, ph = rng.normal(size=modes) / modes, rng.uniform(0, 2 * math.pi, modes)
    return lambda X: sum(a[m] * np.sin(X @ k[m] + ph[m]) for m in range(modes))


def _mesh(dim, n):
    return M.unit_square(n) if dim == 2 else M.unit_cube(n)


def _nodal(mesh, ndof, fn):
    """The piecewise-linear interpolant in an H1 space: vertex dofs first, the rest zero."""
    u = np.zeros(ndof)
    u[:mesh.nv] = fn(mesh.coords)
    return u


def _vertex_wind(rng, mesh):
    """A rotation about a random centre (closed streamlines), sampled at the vertices."""
    c = rng.uniform(0.3, 0.7, mesh.dim)
    Y = mesh.coords - c
    W = np.zeros_like(Y)
    W[:, 0], W[:, 1] = -Y[:, 1], Y[:, 0]
    if mesh.dim == 3:
        W[:, 2] = 0.25
    return W


def _numbers(case, seed):
    """The seed's random numbers, drawn in one order for prepare() and exact()."""
    rng = np.random.default_rng([int(seed), 17])
    f = case['family']
    d = case.get('dim', 2)
    o = dict(rng=rng)
    if f == 'elliptic':
        o.update(diff=float(10 ** rng.uniform(-0.3, 0.3)), src=float(rng.uniform(0.5, 2.0)), g=float(rng.uniform(-1, 1)),
                 dt=case['dt'], u=_field(rng, d))
    elif f in ('transport', 'apply', 'train'):
        o.update(diff=float(10 ** rng.uniform(-2.3, -1.7)), dt=1e-3, u=_field(rng, d))
        w = rng.normal(size=3)
        o['wind'] = tuple(float(x) for x in w[:d] / np.linalg.norm(w[:d]))
    return o


def _form(case, o, wind_dev=None):
    if case['family'] == 'elliptic':
        return fem.make_form(mass=1.0, diff=o['diff'], dt=o['dt']) if o['dt'] else fem.make_form(diff=o['diff'])
    if wind_dev is not None:
        return fem.make_form(mass=1.0, diff=o['diff'], dt=o['dt'], wind_vtx=wind_dev)
    return fem.make_form(mass=1.0, diff=o['diff'], dt=o['dt'], wind=o['wind'])


def prepare(case, seed):
    return {'elliptic': _prepare_elliptic, 'transport': _prepare_transport, 'dg': _prepare_dg, 'direct': _prepare_direct,
            'ins': _prepare_ins, 'batch': _prepare_batch, 'apply': _prepare_apply,
            'train': _prepare_train}[case['family']](case, seed)


def run(state):
    return state['run'](state)


def _prepare_elliptic(case, seed):
    o = _numbers(case, seed)
    mesh = _mesh(case['dim'], case['n'])
    sp = fem.Space(mesh, 'H1', case['order'], mesh.bc_names)
    mixed = case['path'] == 'mixed'
    A = fem.Matrix(sp, fp32=mixed)
    form = _form(case, o)
    b = torch.zeros(sp.ndof, dtype=torch.float64, device='cuda')
    # constant Dirichlet data on the whole boundary; inside, zero (OpenCMP's start of a stationary solve)
    # or the previous step
    u = _nodal(mesh, sp.ndof, o['u']) if o['dt'] else np.zeros(sp.ndof)
    u[np.unique(mesh.bfacets)] = o['g']
    u = _f64(u)
    A.assemble(form)
    sv = fem.KrylovSolver(A, method='CG', precond='jacobi', precision=case['path'], tol=TOL, maxit=20000)
    rhs = fem.make_rhs(dt=o['dt'], src_const=o['src'], mass=1.0, uprev=u) if o['dt'] else fem.make_rhs(src_const=o['src'])
    return dict(run=_run_step, sp=sp, A=A, vals=A.device_values()[0], form=form, rhs=rhs, b=b, u=u, x=torch.zeros_like(b),
                sv=sv)


def _run_step(s):
    s['A'].assemble(s['form'])
    fem.assemble_rhs(s['sp'], s['form'], s['rhs'], s['b'])
    s['sv'].update()
    s['x'].copy_(s['u'])
    s['sv'].solve(s['b'], s['x'])
    return dict(vals=s['vals'], b=s['b'], x=s['x'])


def _prepare_transport(case, seed):
    o = _numbers(case, seed)
    mesh = _mesh(case['dim'], case['n'])
    sp = fem.Space(mesh, 'H1', case['order'], mesh.bc_names)
    W = _f64(_vertex_wind(o['rng'], mesh)) if case['wind'] == 'vertex' else None
    form = _form(case, o, W)
    mixed = case['path'] == 'mixed'
    A = fem.Matrix(sp, jacobi32=True, dfloat=True, sell=True) if mixed else fem.Matrix(sp, jacobi64=True)
    A.assemble(form)
    sv = fem.KrylovSolver(A, method='GMRES', restart=30, precond='jacobi', precision=case['path'],
                          tol=TOL_P3 if case['order'] == 3 else TOL, maxit=2000, inner_tol=1e-4, check_every=6 if mixed else 8)
    u = _nodal(mesh, sp.ndof, o['u'])
    u[~sp.FreeDofs()] = 0.0
    u = _f64(u)
    return dict(run=_run_step, sp=sp, A=A, vals=A.device_values()[0], form=form, W=W, u=u, sv=sv,
                rhs=fem.make_rhs(dt=o['dt'], mass=1.0, uprev=u, dfloat=mixed), b=torch.zeros_like(u),
                x=torch.zeros_like(u))


def _prepare_dg(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    mesh = M.unit_square(case['n'])
    sp = fem.Space(mesh, 'L2', case['order'])
    W = _f64(_vertex_wind(rng, mesh))
    allb = mesh.label_mask(mesh.bc_names)
    form = fem.make_form(mass=1.0, diff=float(10 ** rng.uniform(-3, -2)), dt=2e-3, wind_vtx=W, dg=True, ipc=10.0,
                         nitsche_mask=allb)
    A = fem.Matrix(sp)
    A.assemble(form)
    sv = fem.KrylovSolver(A, method='GMRES', restart=50, precond='block_jacobi', precision='fp64', tol=TOL, maxit=2000)
    fn = _field(rng, 2)
    u = np.zeros((mesh.ne, sp.nloc))
    u[:, 0] = fn(mesh.coords[mesh.elements].mean(1))     # element means: the state a DG run starts from
    u = _f64(u.ravel())
    rhs = fem.make_rhs(dt=2e-3, src_const=float(rng.uniform(0.5, 1.5)), mass=1.0, uprev=u,
                       gval={k: 0.25 * k for k in range(4)})
    return dict(run=_run_step, sp=sp, A=A, vals=A.device_values()[0], form=form, W=W, u=u, sv=sv, rhs=rhs,
                b=torch.zeros_like(u), x=torch.zeros_like(u))


def _prepare_direct(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    mesh = M.unit_square(case['n'])
    sp = fem.Space(mesh, 'L2', case['order'])
    W = _f64(_vertex_wind(rng, mesh))
    form = fem.make_form(mass=1.0, diff=2e-3, dt=5e-2, wind_vtx=W, dg=True, ipc=10.0,
                         nitsche_mask=mesh.label_mask(mesh.bc_names))
    c = rng.uniform(0.25, 0.75, 2)
    fq = _f64(np.exp(-((sp.quad_points() - c) ** 2).sum(-1) / (2 * 0.05 ** 2)))
    A = fem.Matrix(sp)
    A.assemble(form)
    sv = fem.KrylovSolver(A, method='GMRES', restart=50, precond='strip', precision='fp64', tol=TOL, maxit=200)
    sv.strip_gemm(case['gemm'])
    z = torch.zeros(sp.ndof, dtype=torch.float64, device='cuda')
    return dict(run=_run_step, sp=sp, A=A, vals=A.device_values()[0], form=form, W=W, fq=fq, u=z, sv=sv,
                rhs=fem.make_rhs(dt=5e-2, src_qp=fq, gval={k: 0.0 for k in range(4)}), b=torch.zeros_like(z),
                x=torch.zeros_like(z))


def _prepare_ins(case, seed):
    from opencmp_gb300.saddle import SaddleSolver
    rng = np.random.default_rng([int(seed), 17])
    mesh = M.unit_square(case['n'])
    th = fem.TaylorHood(mesh, case['order'], mesh.bc_names)
    A = th.matrix()
    # a vortex that vanishes on the walls, strength and modes from the seed, and a lid whose corners rest
    a, lid = rng.normal(size=(2, 2)), float(rng.uniform(0.5, 1.5))
    X = mesh.coords
    px, py = X[:, 0], X[:, 1]
    u = np.zeros(th.ndof)
    for i in (1, 2):
        for j in (1, 2):
            s, k = a[i - 1, j - 1] / 4, math.pi
            u[:mesh.nv] += s * j * np.sin(i * k * px) ** 2 * np.sin(2 * j * k * py)
            u[th.nu:th.nu + mesh.nv] -= s * i * np.sin(2 * i * k * px) * np.sin(j * k * py) ** 2
    u = _f64(u)
    lab = {q: mesh.bc_names.index(q) for q in mesh.bc_names}
    for comp, val in ((0, lid), (1, 0.0)):
        th.V.set_boundary({lab['top']: val}, th.component(u, comp))
        th.V.set_boundary({lab['bottom']: 0.0, lab['left']: 0.0, lab['right']: 0.0}, th.component(u, comp))
    sv = SaddleSolver(th, A, restart=50, tol=TOL, maxit=1000, precision=case['path'])
    return dict(run=_run_ins, th=th, A=A, u=u, b=torch.zeros_like(u), x=torch.zeros_like(u), sv=sv, dt=1e-3, nu=1e-3)


def _run_ins(s):
    th, dt = s['th'], s['dt']
    th.assemble(s['A'], mass=1.0, nu=s['nu'], dt=dt)
    th.assemble_rhs(s['b'], dt=dt, mass=1.0, uprev=s['u'], imex=s['u'])
    s['sv'].update(mass=1.0, dt=dt, nu=s['nu'])
    s['x'].copy_(s['u'])
    s['sv'].solve(s['b'], s['x'])
    # the constant pressure is fixed by a 1e-10 term alone: a program reads p up to its mean
    p = th.component(s['x'], 2)
    return dict(b=s['b'], u=s['x'][:2 * th.nu], p=p - p.mean())


def _batch_members(case):
    """(n, order, instances) of each member: meshes and orders spread over the range, the count split."""
    top = case['nmax']
    classes = [(max(4, top // d), p) for d in (3, 2, 1) for p in (1, 2, 3)]
    base, extra = divmod(case['count'], len(classes))
    return [(n, p, base + (k < extra)) for k, (n, p) in enumerate(classes) if base + (k < extra)]


def _prepare_batch(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    mem = []
    for n, p, cnt in _batch_members(case):
        mesh = M.unit_square(n)
        sp = fem.Space(mesh, 'H1', p, mesh.bc_names)
        eps, ang = 10 ** rng.uniform(-1, 0, cnt), rng.uniform(0, 2 * math.pi, cnt)
        forms = [fem.make_form(diff=float(e), wind=(math.cos(t), math.sin(t))) for e, t in zip(eps, ang)]
        A = fem.Matrix(sp, batch=cnt, jacobi32=True)
        A.assemble_batch(forms)
        b1 = torch.zeros(sp.ndof, dtype=torch.float64, device='cuda')
        fem.assemble_rhs(sp, forms[0], fem.make_rhs(src_const=1.0), b1)
        sv = fem.KrylovSolver(A, method='GMRES', restart=case['restart'], precision='mixed', tol=TOL, maxit=20000,
                              inner_tol=1e-4)
        mem.append(dict(sp=sp, A=A, forms=forms, sv=sv, b=b1.repeat(cnt),
                        x=torch.zeros(cnt * sp.ndof, dtype=torch.float64, device='cuda')))
    return dict(run=_run_batch, mem=mem, group=fem.KrylovGroup([m['sv'] for m in mem]), bs=[m['b'] for m in mem],
                xs=[m['x'] for m in mem])


def _run_batch(s):
    for m in s['mem']:
        m['A'].assemble_batch(m['forms'])
        m['sv'].update()
        m['x'].zero_()
    s['group'].solve(s['bs'], s['xs'])
    return list(s['xs'])


def _prepare_apply(case, seed):
    o = _numbers(case, seed)
    mesh = _mesh(case['dim'], case['n'])
    sp = fem.Space(mesh, 'H1', case['order'], mesh.bc_names)
    A = fem.Matrix(sp)
    A.assemble(_form(case, o))
    u = _f64(_nodal(mesh, sp.ndof, o['u']))
    return dict(run=_run_apply, sp=sp, A=A, u=u, y=torch.zeros_like(u))


def _run_apply(s):
    s['A'].mult(s['u'], s['y'])
    return s['y']


def _prepare_train(case, seed):
    from opencmp_gb300.guess import LearnedGuess
    o = _numbers(case, seed)
    rng = o['rng']
    mesh = _mesh(case['dim'], case['n'])
    sp = fem.Space(mesh, 'H1', case['order'], mesh.bc_names)
    A = fem.Matrix(sp)
    form = _form(case, o)
    A.assemble(form)
    g = LearnedGuess(sp, k=case['history'], base_order=3, seed=int(seed) & 0xffff)
    p = g.net.params()
    g.net.set_params((p + 0.1 * rng.normal(size=p.size)).astype(np.float32))     # mid-training weights
    d = _field(rng, case['dim'])
    free = _f64(sp.FreeDofs().astype(np.float64))
    u0, u1 = (free * _f64(_nodal(mesh, sp.ndof, f)) for f in (o['u'], d))
    for k in range(case['history'] + 1):
        uk = u0 * math.exp(-0.3 * k) + u1 * math.sin(0.2 * k)
        if k < case['history']:
            g.push(uk)
    b = torch.zeros_like(u0)
    fem.assemble_rhs(sp, form, fem.make_rhs(dt=o['dt'], mass=1.0, uprev=u0), b)
    g.collect(uk, A, b)
    smp = g.samples[0]
    return dict(run=_run_train, g=g, smp=smp, loss=C.c_double(0))


def _run_train(s):
    g, smp = s['g'], s['smp']
    g.net.forward(smp['X'], g.Y)
    LB.call('ocmp_guess_residual_loss', g.net.h, smp['A'].h, fem._ptr(g.Y), fem._ptr(smp['T']), fem._ptr(smp['S']),
            fem._ptr(smp['b']), smp['w'], C.byref(s['loss']), fem._ptr(g.dY), fem._stream(None))
    grad = g.net.backward(smp['X'], g.dY, want_grad=True)
    return dict(Y=g.Y, dY=g.dY, grad=grad)


# ---------------------------------------------------------------- what a pass cannot do without
def _counts(dim, n, order):
    """(elements, vertices, dofs, matrix entries) of the structured H1 space: two dofs share an entry
    when the vertices they live on span a simplex of the mesh."""
    if dim == 2:
        s = [(n + 1) ** 2, 3 * n * n + 2 * n, 2 * n * n, 0]
    else:
        s = [(n + 1) ** 3, 3 * n * (n + 1) ** 2 + 3 * n * n * (n + 1) + n ** 3, 12 * n ** 3 + 6 * n * n, 6 * n ** 3]
    w = {1: 1, 2: order - 1, 3: 1 if order >= 3 else 0, 4: 0}
    comb = lambda a, b: math.comb(a, b) if 0 <= b <= a else 0    # noqa: E731
    nnz = sum(s[k - 1] * sum(w[a] * w[b] * comb(k, a) * comb(a, a + b - k) for a in range(1, k + 1)
                             for b in range(1, k + 1)) for k in range(1, dim + 2))
    return s[dim], s[0], sum(w[k] * s[k - 1] for k in range(1, dim + 2)), nnz


def work(case):
    f, n, p = case['family'], case.get('n', 0), case.get('order', 1)
    if f in ('elliptic', 'transport'):
        # mesh in, matrix values, load vector and solution out, the previous state in; one product
        ne, nv, nd, nnz = _counts(case['dim'], n, p)
        d = case['dim']
        return dict(bytes=4 * (d + 1) * ne + 8 * d * nv + 8 * nnz + 24 * nd, flops=2 * nnz)
    if f == 'apply':
        _, _, nd, nnz = _counts(case['dim'], n, p)
        return dict(bytes=12 * nnz + 20 * nd, flops=2 * nnz)
    if f == 'train':
        # features, target, right-hand side and matrix in (the matrix once more for the transpose),
        # prediction and its gradient out; the network forward and backward
        _, _, nd, nnz = _counts(case['dim'], n, p)
        F = case['history'] - 1
        par = 16 * F + 16 * 16 + 16 * 3 + F
        return dict(bytes=24 * nnz + nd * (4 * F + 28), flops=6 * par * nd + 4 * nnz)
    if f in ('dg', 'direct'):
        L = (p + 1) * (p + 2) // 2
        ne = 2 * n * n
        nnz = L * L * (4 * ne - 4 * n)
        by = 12 * ne + 16 * (n + 1) ** 2 + 8 * nnz + 24 * L * ne
        if f == 'dg':
            return dict(bytes=by, flops=2 * nnz)
        # block elimination over the rows of elements: each strip's inverse formed and applied once
        m = 2 * n * L
        return dict(bytes=by + 2 * 4 * n * m * m, flops=2.0 * n * m ** 3)
    if f == 'ins':
        ne, nv, nu, nnz_u = _counts(2, n, 2)
        nnz = 2 * nnz_u + 4 * 12 * ne
        return dict(bytes=12 * ne + 16 * nv + 8 * nnz + 24 * (2 * nu + nv), flops=2 * nnz)
    by = fl = 0
    for n, p, cnt in _batch_members(case):
        ne, nv, nd, nnz = _counts(2, n, p)
        by += cnt * (8 * nnz + 16 * nd) + 12 * ne + 16 * nv
        fl += cnt * 2 * nnz
    return dict(bytes=by, flops=fl)


# ---------------------------------------------------------------- the same in plain 64-bit torch
def _gauss_simplex(dim, m):
    """Collapsed Gauss-Legendre rule on the reference simplex: points (barycentric), weights."""
    x, w = np.polynomial.legendre.leggauss(m)
    x, w = (x + 1) / 2, w / 2
    g = np.meshgrid(*[x] * dim, indexing='ij')
    gw = np.meshgrid(*[w] * dim, indexing='ij')
    pts, left, wt = [], np.ones_like(g[0]), np.ones_like(g[0])
    for k in range(dim):
        pts.append((g[k] * left).ravel())
        wt = wt * gw[k] * left
        left = left * (1 - g[k])
    lam = np.stack([1 - sum(pts)] + pts, 1)
    return lam, wt.ravel()


def _basis(dim, order, lam):
    """Hierarchical H1 basis (vertex functions, lam_a lam_b and lam_a lam_b (lam_b - lam_a) on edges, face
    bubbles): values (q, L) and derivatives with respect to the barycentric coordinates (q, L, dim + 1)."""
    q, nb = lam.shape[0], dim + 1
    e = np.eye(nb)
    vals, ders = [], []

    def add(v, d):
        vals.append(v)
        ders.append(d)

    for a in range(nb):
        add(lam[:, a], np.broadcast_to(e[a], (q, nb)))
    pairs = [(a, b) for a in range(nb) for b in range(a + 1, nb)]
    if order >= 2:
        for a, b in pairs:
            base = lam[:, a] * lam[:, b]
            dbase = lam[:, [a]] * e[b] + lam[:, [b]] * e[a]
            add(base, dbase)
            if order >= 3:
                t = lam[:, b] - lam[:, a]
                add(base * t, dbase * t[:, None] + base[:, None] * (e[b] - e[a]))
    if order >= 3:
        for a, b in pairs:
            for c in range(b + 1, nb):
                add(lam[:, a] * lam[:, b] * lam[:, c],
                    lam[:, [b]] * lam[:, [c]] * e[a] + lam[:, [a]] * lam[:, [c]] * e[b] + lam[:, [a]] * lam[:, [b]] * e[c])
    return np.stack(vals, 1), np.stack(ders, 1)


def _dofs(dim, order, conn, nv):
    """Vertices, then the edges in ascending (lower, upper) order, then the faces."""
    nb = dim + 1
    cols = [conn]
    at = nv
    pairs = [(a, b) for a in range(nb) for b in range(a + 1, nb)]
    if order >= 2:
        key = torch.stack([conn[:, a] * nv + conn[:, b] for a, b in pairs], 1)
        uniq, inv = torch.unique(key, return_inverse=True)
        for k in range(len(pairs)):
            for m in range(order - 1):
                cols.append(at + inv[:, [k]] * (order - 1) + m)
        at += uniq.numel() * (order - 1)
    if order >= 3:
        tri = [(a, b, c) for a, b in pairs for c in range(b + 1, nb)]
        key = torch.stack([(conn[:, a] * nv + conn[:, b]) * nv + conn[:, c] for a, b, c in tri], 1)
        uniq, inv = torch.unique(key, return_inverse=True)
        cols.append(at + inv)
        at += uniq.numel()
    return torch.cat(cols, 1), at


class _Plain:
    """Matrix and load vector of the H1 cases in 64 bits, by quadrature: torch tensor algebra only."""

    def __init__(self, case):
        mesh = _mesh(case['dim'], case['n'])
        d, order = case['dim'], case['order']
        self.mesh = mesh
        dev = 'cuda'
        conn = torch.as_tensor(np.sort(mesh.elements, 1).astype(np.int64), device=dev)
        X = torch.as_tensor(mesh.coords, device=dev)
        self.dof, self.nd = _dofs(d, order, conn, mesh.nv)
        lam, w = _gauss_simplex(d, order + 2)
        phi, dphi = _basis(d, order, lam)
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)    # noqa: E731
        self.lam, self.w, self.phi, self.dphi = T(lam), T(w), T(phi), T(dphi)
        J = (X[conn[:, 1:]] - X[conn[:, :1]]).transpose(1, 2)
        self.det = torch.linalg.det(J).abs()
        Ji = torch.linalg.inv(J)
        self.gl = torch.cat([-Ji.sum(1, keepdim=True), Ji], 1)       # gradients of the barycentrics (ne, d+1, d)
        self.conn = conn
        free = torch.ones(self.nd, dtype=torch.bool, device=dev)
        bv = T(np.unique(mesh.bfacets))
        onb = torch.zeros(mesh.nv, dtype=torch.bool, device=dev)
        onb[bv] = True
        free[bv] = False
        if order >= 2:
            # a face or edge function is constrained when it lives on a boundary facet
            bf = torch.as_tensor(np.sort(mesh.bfacets, 1).astype(np.int64), device=dev)
            nb = d + 1
            keys = torch.unique(bf[:, 0] * mesh.nv + bf[:, 1] if d == 2 else
                                (bf[:, 0] * mesh.nv + bf[:, 1]) * mesh.nv + bf[:, 2])
            L = self.dof.shape[1]
            for f in range(nb):
                v = [a for a in range(nb) if a != f]
                k = conn[:, v[0]]
                for a in v[1:]:
                    k = k * mesh.nv + conn[:, a]
                hit = torch.isin(k, keys)
                onf = np.array([_lives_on(d, order, i, f) for i in range(L)])
                free[self.dof[hit][:, T(np.flatnonzero(onf))].reshape(-1)] = False
        self.free = free
        self.onb = onb

    def matrix(self, mass=0.0, diff=0.0, dt=1.0, wind=None, wind_vtx=None):
        L = self.dof.shape[1]
        ne = self.dof.shape[0]
        M0 = torch.einsum('q,qi,qj->ij', self.w, self.phi, self.phi)
        S0 = torch.einsum('q,qia,qjb->ijab', self.w, self.dphi, self.dphi)
        G = torch.einsum('ear,ebr->eab', self.gl, self.gl)
        K = dt * diff * torch.einsum('eab,ijab->eij', G, S0) + mass * M0
        if wind_vtx is not None:
            W = torch.as_tensor(wind_vtx, device=K.device)[self.conn]         # ne, d+1, d
            wl = torch.einsum('evr,ear->eva', W, self.gl)
            C0 = torch.einsum('q,qv,qia,qj->ijva', self.w, self.lam, self.dphi, self.phi)
            K -= dt * torch.einsum('eva,ijva->eij', wl, C0)
        elif wind is not None:
            wl = torch.einsum('r,ear->ea', torch.as_tensor(wind, dtype=torch.float64, device=K.device), self.gl)
            C0 = torch.einsum('q,qia,qj->ija', self.w, self.dphi, self.phi)
            K -= dt * torch.einsum('ea,ija->eij', wl, C0)
        K *= self.det[:, None, None]
        row = self.dof[:, :, None].expand(ne, L, L).reshape(-1)
        col = self.dof[:, None, :].expand(ne, L, L).reshape(-1)
        key, inv = torch.unique(row * self.nd + col, return_inverse=True)
        vals = torch.zeros(key.numel(), dtype=torch.float64, device=K.device).index_add_(0, inv, K.reshape(-1))
        r, c = key // self.nd, key % self.nd
        ptr = torch.zeros(self.nd + 1, dtype=torch.int64, device=K.device)
        ptr[1:] = torch.cumsum(torch.bincount(r, minlength=self.nd), 0)
        return torch.sparse_csr_tensor(ptr, c, vals, (self.nd, self.nd)), vals, r == c

    def load(self, dt=1.0, src=0.0, mass=0.0, u=None):
        F = torch.zeros(self.dof.shape, dtype=torch.float64, device=self.det.device)
        if src:
            F += dt * src * torch.einsum('q,qi->i', self.w, self.phi)
        if u is not None:
            M0 = torch.einsum('q,qi,qj->ij', self.w, self.phi, self.phi)
            F += mass * u[self.dof] @ M0
        F *= self.det[:, None]
        return torch.zeros(self.nd, dtype=torch.float64, device=F.device).index_add_(0, self.dof.reshape(-1),
                                                                                      F.reshape(-1))


def _lives_on(d, order, i, f):
    """Whether basis function i is nonzero on the facet lam_f = 0 (sampled at a few of its points)."""
    lam = np.random.default_rng(3).uniform(0.1, 1.0, (4, d + 1))
    lam[:, f] = 0.0
    lam /= lam.sum(1, keepdims=True)
    return bool(np.any(np.abs(_basis(d, order, lam)[0][:, i]) > 1e-14))


def _bicgstab(A, diag, free, b, x):
    """Jacobi-preconditioned BiCGStab with restarts on the true residual, to the floor of 64 bits."""
    f = free.to(b.dtype)
    di = f / torch.where(free, diag, torch.ones_like(diag))
    scale = torch.linalg.vector_norm(f * b) + 1e-300
    for _ in range(6):
        r = f * (b - A @ x)
        if torch.linalg.vector_norm(r) <= 1e-15 * scale:
            break
        rh, rho, p, v, al, om = r.clone(), None, None, None, 1.0, 1.0
        best = torch.linalg.vector_norm(r)
        start = best
        for it in range(3000):
            rho1 = torch.dot(rh, r)
            p = r.clone() if p is None else r + (rho1 / rho) * (al / om) * (p - om * v)
            rho = rho1
            y = di * p
            v = f * (A @ y)
            al = rho / torch.dot(rh, v)
            s = r - al * v
            z = di * s
            t = f * (A @ z)
            om = torch.dot(t, s) / torch.dot(t, t)
            x = x + al * y + om * z
            r = s - om * t
            if it % 10 == 9 and float(torch.linalg.vector_norm(r)) <= 1e-6 * float(start):
                break
    return x


def _cg(A, diag, free, b, x):
    f = free.to(b.dtype)
    di = f / torch.where(free, diag, torch.ones_like(diag))
    for _ in range(4):
        r = f * (b - A @ x)
        n0 = float(torch.linalg.vector_norm(r))
        if n0 <= 1e-15 * float(torch.linalg.vector_norm(f * b)):
            break
        z = di * r
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(4000):
            q = f * (A @ p)
            a = rz / torch.dot(p, q)
            x = x + a * p
            r = r - a * q
            z = di * r
            rz1 = torch.dot(r, z)
            p = z + (rz1 / rz) * p
            rz = rz1
            if it % 20 == 19 and float(torch.linalg.vector_norm(r)) <= 1e-8 * n0:
                break
    return x


def exact(case, seed):
    f = case['family']
    if f not in ('elliptic', 'transport', 'apply'):
        # 'dg', 'direct', 'ins' and 'batch' would need a sparse direct solve in plain torch (their
        # unpreconditioned or point-Jacobi iterations do not get to 64-bit accuracy in time); 'train'
        # is single precision by definition of its network
        return None
    ne, _, _, nnz = _counts(case['dim'], case['n'], case['order'])
    if nnz > 7e7 or ne * {(2, 3): 100, (3, 3): 400}.get((case['dim'], case['order']), 1) > 3e7:
        return None
    o = _numbers(case, seed)
    P = _Plain(case)
    if f == 'elliptic':
        if o['dt']:
            A, vals, isd = P.matrix(1.0, o['diff'], o['dt'])
            x = torch.as_tensor(_nodal(P.mesh, P.nd, o['u']), device='cuda')
        else:
            A, vals, isd = P.matrix(diff=o['diff'])
            x = torch.zeros(P.nd, dtype=torch.float64, device='cuda')
        x[:P.mesh.nv][P.onb] = o['g']
        b = P.load(o['dt'] or 1.0, o['src'], 1.0, x if o['dt'] else None)
        return dict(vals=vals, b=b, x=_cg(A, vals[isd], P.free, b, x))
    u = torch.as_tensor(_nodal(P.mesh, P.nd, o['u']), device='cuda')
    if f == 'apply':
        A, _, _ = P.matrix(mass=1.0, diff=o['diff'], dt=o['dt'], wind=o['wind'])
        return A @ u
    u = torch.where(P.free, u, torch.zeros_like(u))
    if case['wind'] == 'vertex':
        A, vals, isd = P.matrix(1.0, o['diff'], o['dt'], wind_vtx=_vertex_wind(o['rng'], P.mesh))
    else:
        A, vals, isd = P.matrix(1.0, o['diff'], o['dt'], wind=o['wind'])
    b = P.load(mass=1.0, u=u)
    return dict(vals=vals, b=b, x=_bicgstab(A, vals[isd], P.free, b, u.clone()))
