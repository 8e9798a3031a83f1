"""The work that users of this package have it do, as cases to be timed.

A case is a right-hand side of a system, a number of RK45 steps of an
integrator, or one operator apply, through the package's entry points
(``System.rhs``, ``Integrator.run_steps``, ``Backend.kernel('mul', ...)``).
Meshes are periodic boxes: ``uniform``, ``sheared`` (affine cells) or
``bent`` (cells that are not affine), or a mixed box of several element
types.  The forms are plain FP64 (``f64``), FP32 with native operators
(``f32``) and FP32 right-hand sides on the tensor cores under FP64
accumulation (``bf16x3``, the five-product split).

The solution at the start of a case is a smooth random field: a few Fourier
modes of random phase on a mean state of the Mach number that the package's
own test flows have (0.1 for Navier-Stokes, about 1 for Euler).
"""

import math

import numpy as np
import torch

from pyfr_gb300.backend import B200Backend
from pyfr_gb300.cases import euler_mixed, euler_vortex, ns_tgv
from pyfr_gb300.integrators import MixedRKIntegrator, RKVdH2Integrator
from pyfr_gb300.mesh import periodic_box
from pyfr_gb300.solvers.system import EulerSystem, NavierStokesSystem

GAMMA = 1.4
MU, PR = 1.0/1600.0, 0.71           # the Taylor-Green box's gas
TAU = 0.1                           # its LDG penalty


def listed():
    return [
        # The smallest run: the 2-D vortex on 40 x 40 cells, where a step
        # is launches and latency; five steps to a call
        dict(name='vortex40_f64_steps', kind='steps', flow='euler', nd=2,
             n=40, order=3, form='f64', mesh='uniform', rsolver='rusanov',
             beta=0.5, steps=5),
        # One member of the ensemble of vortices at its largest and at its
        # highest order, in the mixed-precision form
        dict(name='vortex96_p4_mixed_steps', kind='steps', flow='euler',
             nd=2, n=96, order=4, form='bf16x3', mesh='uniform',
             rsolver='rusanov', beta=0.5, steps=2),
        # A small Taylor-Green box: a right-hand side that does not fill
        # the chip
        dict(name='tgv8_f64_rhs', kind='rhs', flow='ns', nd=3, n=8, order=3,
             form='f64', mesh='uniform', rsolver='rusanov', beta=0.5,
             steps=0),
        # The Taylor-Green box in FP64, the package's headline workload, at
        # a size whose fields are well beyond the L2 cache
        dict(name='tgv26_f64_rhs', kind='rhs', flow='ns', nd=3, n=26,
             order=3, form='f64', mesh='uniform', rsolver='rusanov',
             beta=0.5, steps=0),
        # The same flow in the mixed-precision form, a whole step (five
        # right-hand sides and stages): the largest case
        dict(name='tgv32_mixed_step', kind='steps', flow='ns', nd=3, n=32,
             order=3, form='bf16x3', mesh='uniform', rsolver='rusanov',
             beta=0.5, steps=1),
        # FP32 throughout, native operators, on affine cells that are not
        # boxes
        dict(name='sheared22_f32_rhs', kind='rhs', flow='ns', nd=3, n=22,
             order=3, form='f32', mesh='sheared', rsolver='rusanov',
             beta=0.5, steps=0),
        # Cells that are not affine, an element count that is no multiple
        # of anything, the other Riemann solver in common use and the
        # central LDG flux, at second order
        dict(name='bent13_p2_f64_rhs', kind='rhs', flow='ns', nd=3, n=13,
             order=2, form='f64', mesh='bent', rsolver='hllc', beta=0.0,
             steps=0),
        # Fourth order in three dimensions: operators larger than one tile
        # of the tensor cores
        dict(name='tgv12_p4_mixed_step', kind='steps', flow='ns', nd=3,
             n=12, order=4, form='bf16x3', mesh='uniform',
             rsolver='rusanov', beta=0.5, steps=1),
        # Hexahedra, pyramids and tetrahedra in one mesh: dense operators
        dict(name='hexpyrtet14_mixed_step', kind='steps', flow='euler',
             nd=3, n=14, order=3, form='bf16x3', mesh='hex-pyr-tet',
             rsolver='rusanov', beta=0.5, steps=1),
        # Euler in FP64 on prisms and hexahedra
        dict(name='hexpri11_f64_rhs', kind='rhs', flow='euler', nd=3, n=11,
             order=3, form='f64', mesh='hex-pri', rsolver='rusanov',
             beta=0.5, steps=0),
        # One operator apply as PyFR's own systems ask for it: the
        # derivative operator of third-order hexahedra in FP64
        dict(name='mul_f64_grad_p3', kind='mul', op='grad', nd=3, order=3,
             form='f64', nvars=5, neles=7001),
        # The same for a dense operator (simplices have no zeros to skip)
        # on the tensor cores
        dict(name='mul_bf16x3_dense', kind='mul', op='dense', nd=3, order=3,
             form='bf16x3', nvars=5, neles=50021),
    ]


def draw(rng):
    """One more case of the ranges of the listed ones."""
    def between(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    what = rng.choice(['vortex', 'tgv', 'tgv', 'tgv', 'mixed', 'mul'])
    form = rng.choice(['f64', 'bf16x3', 'f32'])
    if what == 'vortex':
        order = rng.choice([2, 3, 4])
        if form == 'f32':
            form = 'f64'
        return dict(kind='steps', flow='euler', nd=2, n=between(16, 97),
                    order=order, form=form,
                    mesh=rng.choice(['uniform', 'sheared']),
                    rsolver='rusanov', beta=0.5, steps=rng.choice([1, 2, 5]))
    if what == 'tgv':
        order = rng.choice([2, 3, 3, 4])
        hi = {2: 24, 3: 22, 4: 13}[order]
        steps = rng.choice([0, 1]) if form != 'bf16x3' else 1
        return dict(kind='steps' if steps else 'rhs', flow='ns', nd=3,
                    n=between(5, hi), order=order,
                    form='f64' if steps and form == 'f32' else form,
                    mesh=rng.choice(['uniform', 'uniform', 'sheared',
                                     'bent']),
                    rsolver='rusanov' if steps else
                    rng.choice(['rusanov', 'hllc']),
                    beta=rng.choice([0.5, 0.5, -0.5, 0.0]), steps=steps)
    if what == 'mixed':
        if form == 'f32':
            form = 'bf16x3'
        steps = 1 if form == 'bf16x3' else 0
        return dict(kind='steps' if steps else 'rhs', flow='euler', nd=3,
                    n=2*between(2, 6), order=rng.choice([2, 3]), form=form,
                    mesh=rng.choice(['hex-pri', 'pri-tet', 'hex-pyr-tet']),
                    rsolver='rusanov', beta=0.5, steps=steps)
    return dict(kind='mul', op=rng.choice(['grad', 'interp', 'lift',
                                           'dense']),
                nd=3, order=rng.choice([2, 3]), form=form,
                nvars=5, neles=between(200, 30000))


# ---- one-dimensional operators of the Gauss-Legendre elements -------------

def _line(order):
    """Points, weights, differentiation matrix and the values of the
    Lagrange basis at -1 and +1."""
    x, w = np.polynomial.legendre.leggauss(order + 1)
    c = np.array([1/np.prod(x[j] - np.delete(x, j)) for j in range(len(x))])
    D = np.zeros((len(x),)*2)
    for i in range(len(x)):
        for j in range(len(x)):
            if i != j:
                D[i, j] = c[j]/c[i]/(x[i] - x[j])
        D[i, i] = -D[i].sum()
    ends = [np.array([np.prod(e - np.delete(x, j))*c[j]
                      for j in range(len(x))]) for e in (-1.0, 1.0)]
    return x, w, D, ends[0], ends[1]


def _operator(case):
    """The matrix of a 'mul' case (rows x columns)."""
    x, w, D, lo, hi = _line(case['order'])
    n, nd = len(x), case['nd']
    eye = np.eye(n)
    if case['op'] == 'dense':
        # (rows and columns of a tetrahedron's face lift: every flux point
        # reaches every solution point)
        p = case['order']
        m, k = (p + 1)*(p + 2)*(p + 3)//6, 4*(p + 1)*(p + 2)//2
        i, j = np.mgrid[:m, :k]
        return np.cos(1.0 + 0.7*i + 0.37*i*j + 0.11*j)

    def kron(mats):
        # (the first coordinate is the fastest)
        out = np.eye(1)
        for a in mats:
            out = np.kron(a, out)
        return out

    if case['op'] == 'grad':
        return np.vstack([kron([D if e == d else eye for e in range(nd)])
                          for d in range(nd)])
    if case['op'] == 'lift':
        lo, hi = lo/w, hi/w
    a = np.vstack([kron([v[None] if e == d else eye for e in range(nd)])
                   for d in range(nd) for v in (lo, hi)])
    return a if case['op'] == 'interp' else a.T


# ---- inputs ------------------------------------------------------------------

def _field(case, seed, coords):
    """Conserved variables (nvars, *shape) at logical coordinates (a list of
    nd arrays in [0, 2 pi))."""
    rng = np.random.default_rng([seed, 11])
    nd = case['nd']
    if case['flow'] == 'ns':
        rho0, p0, v0, amp = 1.0, 1/(GAMMA*0.01), [0.0]*nd, 0.5
    else:
        rho0, p0, v0, amp = 1.0, 1.0, [1.0, 0.5, 0.25][:nd], 0.2

    def modes():
        out = np.zeros(np.broadcast_shapes(*[c.shape for c in coords]))
        for _ in range(3):
            k = rng.integers(1, 3, nd)
            s = rng.uniform(0, 2*np.pi, nd)
            term = rng.uniform(0.4, 1.0)
            for c, kk, ss in zip(coords, k, s):
                term = term*np.sin(kk*c + ss)
            out = out + term
        return out

    # (perturbations of pressure and density as a flow of this velocity
    # makes them)
    m2 = amp*amp*rho0
    v = [v0[d] + amp*modes() for d in range(nd)]
    p = p0 + 0.3*m2*modes()
    rho = rho0*(1 + 0.3*m2/(GAMMA*p0)*modes()) if case['flow'] == 'ns' else \
        rho0*(1 + 0.1*modes())
    E = p/(GAMMA - 1) + 0.5*rho*sum(c*c for c in v)
    return np.stack([rho] + [rho*c for c in v] + [E])


def _half(case):
    """Half-width of the undeformed box."""
    return 10.0 if case['nd'] == 2 else math.pi


def _deform(case, x):
    """The mesh's vertices from those of the uniform box: x (..., nd)."""
    nd, half = case['nd'], _half(case)
    if case['mesh'] == 'uniform':
        return x
    y = x.copy()
    if case['mesh'] == 'sheared':
        y[..., 0] = x[..., 0] + 0.3*x[..., 1]
        if nd == 3:
            y[..., 1] = x[..., 1] - 0.2*x[..., 2]
    else:
        s = math.pi/half
        for d in range(nd):
            y[..., d] += 0.08/s*np.sin(s*x[..., (d + 1) % nd] + 0.3)* \
                np.cos(s*x[..., d])
    return y


def _config(case):
    single = case['form'] != 'f64'
    prec = 'single' if single else 'double'
    if case['mesh'] in ('hex-pri', 'pri-tet', 'hex-pyr-tet'):
        cfg, mesh = euler_mixed(n=case['n'], order=case['order'],
                                kinds=case['mesh'], precision=prec)
    elif case['flow'] == 'euler':
        cfg, mesh = euler_vortex(n=case['n'], order=case['order'], dt=1e-3,
                                 rsolver=case['rsolver'], precision=prec)
    else:
        cfg, mesh = ns_tgv(n=case['n'], order=case['order'], dt=5e-4,
                           rsolver=case['rsolver'], beta=case['beta'],
                           tau=TAU, precision=prec)
    if case['mesh'] in ('sheared', 'bent'):
        for et in mesh.spts:
            mesh.spts[et] = _deform(case, mesh.spts[et])
    if case['form'] == 'bf16x3':
        cfg.set('backend-b200', 'mul-precision', 'bf16x3')
        cfg.set('backend-b200', 'split-products', '5')
    return cfg, mesh


def _logical(case):
    """Logical coordinates of the solution points of a box in the order of
    the solution arrays: nd arrays (nupts, neles)."""
    nd, n = case['nd'], case['n']
    x = _line(case['order'])[0]
    pts = np.meshgrid(*[x]*nd, indexing='ij')[::-1]      # first is fastest
    ele = np.indices((n,)*nd)[::-1]
    return [2*np.pi/n*(e.reshape(1, -1) + 0.5*(1 + p.reshape(-1, 1)))
            for e, p in zip(ele, pts)]


class _View:
    """Device memory of the package as an array of torch's."""

    def __init__(self, m):
        shape = m.datashape[1:]
        self.__cuda_array_interface__ = dict(
            shape=tuple(int(s) for s in shape), typestr=m.dtype.str,
            data=(int(m.data), False), version=3)


def _tensor(m):
    return torch.as_tensor(_View(m), device='cuda')


def _prepare_mul(case, seed):
    cfg, _ = _config(dict(case, n=2, mesh='uniform', flow='ns',
                          rsolver='rusanov', beta=0.5))
    be = B200Backend(cfg)
    a = _operator(case)
    am = be.const_matrix(a, tags={'align'})
    shape = (case['nvars'], case['neles'])
    b = be.matrix((a.shape[1],) + shape, tags={'align'})
    out = be.matrix((a.shape[0],) + shape, tags={'align'})
    be.commit()
    g = torch.Generator(device='cuda').manual_seed(seed)
    _tensor(b).copy_(_mul_input(case, a.shape[1], g))
    torch.cuda.synchronize()
    k = be.kernel('mul', am, b, out)
    be.run_kernels([k], wait=True)
    return dict(kind='mul', be=be, k=k, keep=(am, b, out),
                out=[_tensor(out)])


def _mul_input(case, rows, g):
    """The columns of one variable of one element vary smoothly about a
    mean, each variable with its own scale."""
    nb = -(-case['neles']//32)
    dev = g.device
    dt = torch.float64
    scale = torch.tensor([1.0, 0.5, 0.5, 0.5, 20.0], dtype=dt, device=dev)
    mean = torch.tensor([1.0, 0.1, 0.0, -0.1, 150.0], dtype=dt, device=dev)
    r = torch.linspace(0, 1, rows, dtype=dt, device=dev)[:, None, None, None]
    ph = torch.rand((2, 1, nb, case['nvars'], 32), generator=g, dtype=dt,
                    device=dev)
    v = mean[:, None] + scale[:, None]*(torch.sin(6*ph[0] + 3*r) +
                                        0.3*torch.cos(9*ph[1] + 8*r))
    # (the padding of the last block of elements is zero)
    e = torch.arange(nb*32, device=dev).reshape(nb, 1, 32)
    v = torch.where(e < case['neles'], v, torch.zeros((), dtype=dt,
                                                      device=dev))
    return v.to(torch.float64 if case['form'] == 'f64' else torch.float32)


def prepare(case, seed):
    if case['kind'] == 'mul':
        return _prepare_mul(case, seed)
    cfg, mesh = _config(case)
    be = B200Backend(cfg)
    cls = EulerSystem if case['flow'] == 'euler' else NavierStokesSystem

    if case['mesh'] in ('hex-pri', 'pri-tet', 'hex-pyr-tet'):
        # (the solution at the points of every element type)
        probe = cls(B200Backend(cfg), mesh, None, 1, cfg)
        init = {}
        for et, p in zip(probe.ele_types, probe.ele_ploc_upts):
            c = [np.ascontiguousarray(p[:, d]) for d in range(3)]
            init[et] = _field(case, seed, c).swapaxes(0, 1)
    else:
        et = next(iter(mesh.spts))
        init = {et: _field(case, seed, _logical(case)).swapaxes(0, 1)}

    if case['kind'] == 'rhs':
        s = cls(be, mesh, init, 2, cfg)
        s.commit()
        return dict(kind='rhs', be=be, sys=s,
                    out=[_tensor(b[1]) for b in s.ele_banks])

    icls = MixedRKIntegrator if case['form'] == 'bf16x3' else RKVdH2Integrator
    intg = icls(be, cls, mesh, cfg, init)
    return dict(kind='steps', be=be, intg=intg, steps=case['steps'],
                mixed=case['form'] == 'bf16x3')


def run(state):
    if state['kind'] == 'mul':
        state['be'].run_kernels([state['k']])
        return state['out']
    if state['kind'] == 'rhs':
        state['sys'].rhs(0.0, 0, 1)
        return state['out']
    intg = state['intg']
    intg.run_steps(state['steps'])
    # The solution: the FP64 accumulators of the mixed form, the current
    # register of the plain one
    if state['mixed']:
        return [_tensor(m) for m in intg.acc]
    return [_tensor(b[intg.idxcurr]) for b in intg.system.ele_banks]


# ---- what a pass cannot do without --------------------------------------------

def _npts(case):
    """(solution points, face points, nonzeros of all operator applies of a
    right-hand side and variable) summed over the elements."""
    p, nd, n = case['order'], case['nd'], case['n']
    q = p + 1
    tri, quad = q*(q + 1)//2, q*q
    tet, pri, pyr = q*(q + 1)*(q + 2)//6, tri*q, q*(q + 1)*(2*q + 1)//6
    if case['mesh'] in ('uniform', 'sheared', 'bent'):
        ne, nu, nf = n**nd, q**nd, 2*nd*q**(nd - 1)
        # interpolation, derivatives with corrections, divergence
        nnz = nf*q + nd*nu*(q + 2)
        if case['flow'] == 'ns':
            nnz += nd*nu*(q + 2) + nd*nf*q
        return ne*nu, ne*nf, ne*nnz
    h = n**3//2
    kinds = {'hex-pri': [(h, q**3, 6*quad, 1), (2*h, pri, 3*quad + 2*tri, 0)],
             'pri-tet': [(2*h, pri, 3*quad + 2*tri, 0), (6*h, tet, 4*tri, 0)],
             # one pyramid per face between the halves, the rest tetrahedra
             'hex-pyr-tet': [(h, q**3, 6*quad, 1),
                             (2*n*n, pyr, quad + 4*tri, 0),
                             (2*(6*h - 2*n*n), tet, 4*tri, 0)]}[case['mesh']]
    nu = sum(e*u for e, u, f, t in kinds)
    nf = sum(e*f for e, u, f, t in kinds)
    nnz = sum(e*((f*q + 3*u*(q + 2)) if t else (f*u + 3*u*u + u*f))
              for e, u, f, t in kinds)
    return nu, nf, nnz


def work(case):
    isz = 8 if case['form'] == 'f64' else 4
    if case['kind'] == 'mul':
        a = _operator(case)
        ncol = case['nvars']*case['neles']
        return dict(bytes=(a.shape[0] + a.shape[1])*ncol*isz,
                    flops=2.0*int(np.count_nonzero(np.abs(a) > 1e-14))*ncol)
    nv = case['nd'] + 2
    nu, nf, nnz = _npts(case)
    ns = case['flow'] == 'ns'
    flops = 2.0*nnz*nv + nu*(200 if ns else 60) + 0.5*nf*(200 if ns else 90)
    if case['kind'] == 'rhs':
        return dict(bytes=2*nu*nv*isz, flops=flops)
    # (a step cannot keep its registers on the chip: each of the five stages
    # reads and writes the solution, and the input of its right-hand side)
    state = nu*nv*8
    return dict(bytes=case['steps']*5*(2*state + 2*nu*nv*isz),
                flops=case['steps']*5*(flops + 4*nu*nv))


# ---- the same in 64 bits, with torch alone ---------------------------------------

class _Box:
    """Flux reconstruction on a periodic box of quadrilaterals or
    hexahedra.  Fields are (nvars, cells z..x, points z..x); the face on
    the high side of a cell is its interface's left one."""

    def __init__(self, case, dev):
        self.case, self.dev = case, dev
        self.nd, self.n = case['nd'], case['n']
        x, w, D, lo, hi = _line(case['order'])
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
        self.D, self.lo, self.hi = t(D), t(lo), t(hi)
        self.glo, self.ghi = t(lo/w), t(hi/w)
        q = len(x)
        # Vertices (2, .., 2 (z..x), cells z..x, nd)
        half, n = _half(case), self.n
        ax = np.linspace(-half, half, n + 1)
        nd = self.nd
        verts = np.empty((2,)*nd + (n,)*nd + (nd,))
        for v in np.ndindex(*(2,)*nd):
            g = np.meshgrid(*[ax[o:o + n] for o in v], indexing='ij')
            verts[v] = np.stack(g[::-1], -1)
        verts = _deform(case, verts)
        self.S, self.det = self._metrics(verts, [x]*nd)
        self.Sf = [[self._metrics(verts, [np.array([e]) if f == d else x
                                          for f in range(nd)])[0]
                    for e in (-1.0, 1.0)] for d in range(nd)]
        self.q = q

    def _metrics(self, verts, pts):
        """S[i][j] and |J| at the product of the lines pts (x first)."""
        nd = self.nd
        J = {}
        for i in range(nd):
            ops = []
            for d in range(nd):
                p = pts[d]
                ops.append(np.stack([-0.5 + 0*p, 0.5 + 0*p], 1) if d == i
                           else np.stack([0.5*(1 - p), 0.5*(1 + p)], 1))
            a = verts                                  # (2 z..x, cells, nd)
            for d in range(nd):
                # contract the vertex axis of direction d (axis nd-1-d)
                a = np.moveaxis(np.tensordot(ops[d], a, (1, nd - 1 - d)),
                                0, nd - 1 - d)
            a = np.moveaxis(a, list(range(nd)), list(range(nd, 2*nd)))
            for j in range(nd):
                J[i, j] = torch.tensor(np.ascontiguousarray(a[..., j]),
                                       device=self.dev)
        if nd == 2:
            S = [[J[1, 1], -J[1, 0]], [-J[0, 1], J[0, 0]]]
        else:
            S = []
            for i in range(3):
                a, b = (i + 1) % 3, (i + 2) % 3
                S.append([J[a, 1]*J[b, 2] - J[a, 2]*J[b, 1],
                          J[a, 2]*J[b, 0] - J[a, 0]*J[b, 2],
                          J[a, 0]*J[b, 1] - J[a, 1]*J[b, 0]])
        det = sum(J[0, j]*S[0][j] for j in range(nd))
        return S, det

    # (axes counted from the end: points x is -1, cells x is -1 - nd)
    def apply(self, op, u, d):
        """op (m, q) along the points of direction d."""
        return torch.movedim(torch.tensordot(u, op, ([u.dim() - 1 - d], [1])),
                             -1, u.dim() - 1 - d)

    def ends(self, u, d):
        return self.apply(self.lo[None], u, d), self.apply(self.hi[None], u,
                                                           d)

    def lift(self, g, v, d):
        """Face values (one point in direction d) times g along d."""
        shape = [1]*v.dim()
        shape[v.dim() - 1 - d] = len(g)
        return v*g.reshape(shape)

    def nb(self, v, d):
        """The value of the next cell in direction d."""
        return torch.roll(v, -1, v.dim() - 1 - self.nd - d)

    def back(self, v, d):
        return torch.roll(v, 1, v.dim() - 1 - self.nd - d)

    def inviscid(self, u):
        nd = self.nd
        v = [u[1 + i]/u[0] for i in range(nd)]
        p = (GAMMA - 1)*(u[-1] - 0.5*sum(u[1 + i]*v[i] for i in range(nd)))
        f = [torch.stack([u[1 + i]] + [u[1 + j]*v[i] + (p if i == j else 0)
                                       for j in range(nd)] +
                         [(u[-1] + p)*v[i]]) for i in range(nd)]
        return f, v, p

    def viscous(self, u, g):
        nd, rho = self.nd, u[0]
        v = [u[1 + i]/rho for i in range(nd)]
        dv = [[(g[d][1 + i] - v[i]*g[d][0])/rho for d in range(nd)]
              for i in range(nd)]
        div = sum(dv[i][i] for i in range(nd))
        out = []
        for d in range(nd):
            dT = (g[d][-1] - g[d][0]*u[-1]/rho)/rho - \
                sum(v[i]*dv[i][d] for i in range(nd))
            tau = [-MU*(dv[i][d] + dv[d][i] - (2.0/3.0*div if i == d else 0))
                   for i in range(nd)]
            out.append(torch.stack([torch.zeros_like(rho)] + tau +
                                   [sum(v[i]*tau[i] for i in range(nd)) -
                                    MU*GAMMA/PR*dT]))
        return out

    def riemann(self, ul, ur, nrm):
        nd = self.nd
        fl, vl, pl = self.inviscid(ul)
        fr, vr, pr = self.inviscid(ur)
        fln = sum(nrm[d]*fl[d] for d in range(nd))
        frn = sum(nrm[d]*fr[d] for d in range(nd))
        nvl = sum(nrm[d]*vl[d] for d in range(nd))
        nvr = sum(nrm[d]*vr[d] for d in range(nd))
        if self.case['rsolver'] == 'rusanov':
            a = torch.sqrt(GAMMA*(pl + pr)/(ul[0] + ur[0])) + \
                0.5*torch.abs(nvl + nvr)
            return 0.5*(fln + frn) + 0.5*a*(ul - ur)
        # HLLC with Roe averages for the wave speeds
        sl_, sr_ = torch.sqrt(ul[0]), torch.sqrt(ur[0])
        inv = 1/(sl_ + sr_)
        nv = (sl_*nvl + sr_*nvr)*inv
        H = (sl_*(pr + ur[-1]) + sr_*(pl + ul[-1]))/(sl_*ur[0] + sr_*ul[0])
        qq = sum(((vl[d]*sl_ + vr[d]*sr_)*inv)**2 for d in range(nd))
        a = torch.sqrt((GAMMA - 1)*(H - 0.5*qq))
        sl = torch.minimum(nv - a, nvl - torch.sqrt(GAMMA*pl/ul[0]))
        sr = torch.maximum(nv + a, nvr + torch.sqrt(GAMMA*pr/ur[0]))
        ss = (pr - pl + ul[0]*nvl*(sl - nvl) - ur[0]*nvr*(sr - nvr)) / \
            (ul[0]*(sl - nvl) - ur[0]*(sr - nvr))

        def star(u, v, nvk, pk, sk):
            c = (sk - nvk)/(sk - ss)
            r = c*u[0]
            return torch.stack([r] + [r*(v[d] + (ss - nvk)*nrm[d])
                                      for d in range(nd)] +
                               [c*(u[-1] + (ss - nvk)*(u[0]*ss +
                                                       pk/(sk - nvk)))])
        fsl = fln + sl*(star(ul, vl, nvl, pl, sl) - ul)
        fsr = frn + sr*(star(ur, vr, nvr, pr, sr) - ur)
        return torch.where(sl >= 0, fln, torch.where(
            ss >= 0, fsl, torch.where(sr >= 0, fsr, frn)))

    def rhs(self, u):
        nd, beta = self.nd, self.case['beta']
        ns = self.case['flow'] == 'ns'
        uf = [self.ends(u, d) for d in range(nd)]
        if ns:
            gt = []
            for d in range(nd):
                l, r = uf[d][1], self.nb(uf[d][0], d)
                c = (0.5 + beta)*r + (0.5 - beta)*l
                gt.append(self.apply(self.D, u, d) +
                          self.lift(self.ghi, c - l, d) -
                          self.lift(self.glo, self.back(c, d) - uf[d][0], d))
            g = [sum(self.S[k][i]*gt[k] for k in range(nd))/self.det
                 for i in range(nd)]
        f = self.inviscid(u)[0]
        if ns:
            f = [a + b for a, b in zip(f, self.viscous(u, g))]
        out = 0
        for d in range(nd):
            ft = sum(self.S[d][k]*f[k] for k in range(nd))
            lo, hi = self.ends(ft, d)
            l, r = uf[d][1], self.nb(uf[d][0], d)
            nrm = self.Sf[d][1][d]
            mag = torch.sqrt(sum(x*x for x in nrm))
            nrm = [x/mag for x in nrm]
            fc = self.riemann(l, r, nrm)
            if ns:
                for wt, side, k in ((0.5 + beta, l, 1), (0.5 - beta, r, 0)):
                    if not wt:
                        continue
                    gf = [self.ends(x, d)[k] for x in g]
                    gf = gf if k else [self.nb(x, d) for x in gf]
                    fv = self.viscous(side, gf)
                    fc = fc + wt*sum(nrm[j]*fv[j] for j in range(nd))
                fc = fc + TAU*(l - r)
            fc = mag*fc
            out = out + self.apply(self.D, ft, d) + \
                self.lift(self.ghi, fc - hi, d) - \
                self.lift(self.glo, self.back(fc, d) - lo, d)
        return -out/self.det

    def pack(self, u):
        """(nvars, cells, points) to the package's arrays, padded."""
        nd, nv = self.nd, self.nd + 2
        ne, nu = self.n**nd, self.q**nd
        a = u.reshape(nv, ne, nu).permute(2, 0, 1)
        nb = -(-ne//32)
        a = torch.nn.functional.pad(a, (0, nb*32 - ne))
        return a.reshape(nu, nv, nb, 32).permute(0, 2, 1, 3).contiguous()


RK_A = [970286171893/4311952581923, 6584761158862/12103376702013,
        2251764453980/15575788980749, 26877169314380/34165994151039]
RK_B = [1153189308089/22510343858157, 1772645290293/4653164025191,
        -1672844663538/4480602732383, 2114624349019/3568978502595,
        5198255086312/14908931495163]


def exact(case, seed):
    dev = torch.device('cuda' if torch.cuda.is_available() else 'cpu')
    if case['kind'] == 'mul':
        a = torch.tensor(_operator(case), dtype=torch.float64, device=dev)
        g = torch.Generator(device=dev).manual_seed(seed)
        b = _mul_input(case, a.shape[1], g).to(torch.float64)
        return [torch.tensordot(a, b, 1)]
    if case['mesh'] in ('hex-pri', 'pri-tet', 'hex-pyr-tet'):
        # (the operators and points of prisms, pyramids and tetrahedra are
        # tables of the package)
        return None
    box = _Box(case, dev)
    nd, n, q = case['nd'], case['n'], box.q
    u = _field(case, seed, _logical(case))              # (nv, nupts, neles)
    if case['kind'] == 'rhs' and case['form'] != 'f64':
        u = u.astype(np.float32).astype(np.float64)
    u = torch.tensor(u, device=dev).permute(0, 2, 1).contiguous()
    u = u.reshape((nd + 2,) + (n,)*nd + (q,)*nd)
    if case['kind'] == 'rhs':
        return [box.pack(box.rhs(u))]

    x = y = u
    dt = 1e-3 if case['flow'] == 'euler' else 5e-4
    for _ in range(case['steps']):
        y = x
        for i in range(5):
            r = box.rhs(y)
            if i < 4:
                y = x + RK_A[i]*dt*r
            x = x + RK_B[i]*dt*r
    if case['form'] == 'bf16x3' and case['rsolver'] == 'rusanov':
        # The mixed form accumulates the perturbation from the mean state,
        # its energy less the mean enthalpy times the density's
        dims = list(range(1, u.dim()))
        p = (GAMMA - 1)*(u[-1] - 0.5*(u[1:-1]**2).sum(0)/u[0])
        rho, mom, p = u[0].mean(), u[1:-1].mean(dims), p.mean()
        if case['flow'] == 'ns':
            mom = mom*0
        E = p/(GAMMA - 1) + 0.5*(mom**2).sum()/rho
        ref = torch.cat([rho[None], mom, E[None]])
        x = x - ref.reshape([-1] + [1]*(x.dim() - 1))
        x = torch.cat([x[:-1], (x[-1] - (E + p)/rho*x[0])[None]])
    return [box.pack(x)]
