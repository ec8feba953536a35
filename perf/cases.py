"""Performance cases of the sparse solver: what a finite-element program has the library do.

Every mesh is an n^3 box of unit hex8 elements (3 DOF per node, face x = 0 clamped), the
sizes being those whose symbolic structures the package ships.  A case is one of

  factor_solve  assemble SM from element moduli, K - sigma M when shifted, factor, solve
  mixed         the same in the mixed-precision mode, refined to a backward error of 1e-13
  solve         sweeps on a factor that is already there
  batch         many independent shifted systems factored and solved as one forest
  adjoint       forward solve and gradient of a SIMP-parametrised stiffness
  sprsol        the Fortran entry point on page-locked host arrays
  assemble      hex8 element matrices of a distorted mesh, assembled into SM

Structures, element topologies and host control arrays depend on the mesh alone and are kept
for the process, as a program with one mesh keeps them.  The solver handle (plan and device
buffers) is made in prepare().
"""
import functools
import math

import numpy as np
import torch

import sam_lib_b200 as spr
from sam_lib_b200 import adjoint, batch, system

SIZES = (3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 16, 20, 24, 32, 48)
LAMBDA1_N2 = 0.4476          # lowest eigenvalue of (K, M) with E = 1, times n^2


def listed():
    return [
        # a large static analysis: four load cases on 346k equations
        dict(name='box48_rhs4', kind='factor_solve', n=48, nrhs=4, decades=1.0, shift=0.0, rule='ldl'),
        # a frequency response: K - sigma M above the first modes, one load case
        dict(name='box32_shifted_rhs1', kind='factor_solve', n=32, nrhs=1, decades=0.5, shift=2.5, rule='ldl'),
        # the factorisation that shift-invert Lanczos calls (SPRFC3), and its first solve
        dict(name='box20_fc3_rhs1', kind='factor_solve', n=20, nrhs=1, decades=0.5, shift=2.5, rule='replace'),
        # the usual component model
        dict(name='box12_rhs3', kind='factor_solve', n=12, nrhs=3, decades=1.5, shift=0.0, rule='ldl'),
        # the smallest: a substructure of a few hundred equations, all latency
        dict(name='box4_rhs1', kind='factor_solve', n=4, nrhs=1, decades=0.5, shift=0.0, rule='ldl'),
        # mixed precision with refinement in place of an FP64 factorisation
        dict(name='box32_mixed_rhs4', kind='mixed', n=32, nrhs=4, decades=0.5),
        # a Lanczos step: SPRFS1 then SPRBS1 on one vector
        dict(name='solve32_split_rhs1', kind='solve', n=32, nrhs=1, decades=1.0, sweeps='split'),
        # many load cases on a stored factor
        dict(name='solve24_rhs40', kind='solve', n=24, nrhs=40, decades=1.0, sweeps='both'),
        # 512 uneven shifted systems, 16 right-hand sides each
        dict(name='batch512_rhs16', kind='batch', count=512, sizes=3, nrhs=16),
        # a topology optimisation step
        dict(name='adjoint32', kind='adjoint', n=32, nrhs=1),
        # a Fortran program's SPRSOL on its own arrays
        dict(name='sprsol20_rhs4', kind='sprsol', n=20, nrhs=4, decades=1.0),
        # a nonlinear analysis forming its tangent stiffness
        dict(name='assemble32', kind='assemble', n=32, amp=0.15),
    ]


def draw(rng):
    def size(most, least=3):
        return rng.choice([n for n in SIZES if least <= n <= most])

    def nrhs(most):
        return min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1)))))

    decades = round(rng.uniform(0.2, 1.6), 2)
    kind = rng.choice(['factor_solve', 'factor_solve', 'factor_solve', 'mixed', 'solve', 'solve', 'batch', 'adjoint',
                       'sprsol', 'assemble'])
    if kind == 'factor_solve':
        shift = rng.choice([0.0, round(rng.uniform(0.3, 4.0), 2)])
        return dict(kind=kind, n=size(32), nrhs=nrhs(20), decades=decades, shift=shift,
                    rule=rng.choice(['ldl', 'ldl', 'replace']))
    if kind == 'mixed':
        return dict(kind=kind, n=size(32, 12), nrhs=nrhs(8), decades=round(rng.uniform(0.1, 0.6), 2))
    if kind == 'solve':
        return dict(kind=kind, n=size(32), nrhs=nrhs(48), decades=decades,
                    sweeps=rng.choice(['both', 'split', 'forward', 'back']))
    if kind == 'batch':
        return dict(kind=kind, count=int(16 * 2 ** rng.uniform(0.0, 5.0)), sizes=rng.randrange(1000), nrhs=nrhs(16))
    if kind == 'adjoint':
        return dict(kind=kind, n=size(32, 5), nrhs=nrhs(6))
    if kind == 'sprsol':
        return dict(kind=kind, n=size(20), nrhs=nrhs(12), decades=decades)
    return dict(kind=kind, n=size(32), amp=round(rng.uniform(0.02, 0.2), 3))


# ---- what depends on the mesh alone

@functools.lru_cache(maxsize=None)
def _system(n):
    return system.HexSystem(n)


@functools.lru_cache(maxsize=None)
def _elements(n):
    return adjoint.ElementOps(_system(n))


@functools.lru_cache(maxsize=None)
def _mass(n):
    """(diagonal positions in SM, lumped mass per equation)."""
    hs = _system(n)
    return system.diag_positions(hs.mspar, hs.mtrees, hs.msifa), hs.to_internal(hs.box.lumped_mass())


@functools.lru_cache(maxsize=None)
def _mesh(n):
    """(diagonal positions in SM, lumped mass per equation, element matrix) on the device."""
    ke = np.asfortranarray(_system(n).ke).ravel(order='F').copy()
    return tuple(torch.from_numpy(a).cuda() for a in _mass(n) + (ke,))


@functools.lru_cache(maxsize=None)
def _unit_sm(n):
    return _system(n).assemble()


def _batch_sizes(case):
    return [int(v) for v in np.random.default_rng(case['sizes']).integers(3, 13, size=case['count'])]


# ---- inputs

def _moduli(case, seed):
    """Element moduli, log-uniform over the case's decades below 1."""
    g = np.random.default_rng([seed, 1])
    return 10.0 ** g.uniform(-case['decades'], 0.0, size=_system(case['n']).box.nel)


def _loads(case, seed):
    g = np.random.default_rng([seed, 2])
    return g.uniform(-1.0, 1.0, size=(case['nrhs'], _system(case['n']).neq))


def _sigma(case):
    return case.get('shift', 0.0) * LAMBDA1_N2 / case['n'] ** 2 * 10.0 ** (-0.5 * case['decades'])


def _batch_draws(case, seed):
    g = np.random.default_rng([seed, 3])
    fac = g.uniform(0.5, 2.0, size=case['count'])
    ns = _batch_sizes(case)
    sigma = [f * LAMBDA1_N2 / n ** 2 for f, n in zip(fac, ns)]
    return ns, sigma, [g.uniform(-1.0, 1.0, size=(case['nrhs'], _system(n).neq)) for n in ns]


def _assembled(st, sm):
    """SM = K (- sigma M), assembled on the device from the element moduli."""
    n = st['n']
    pos, mass, ke = _mesh(n)
    _elements(n).assemble(sm, ke, st['moduli'])
    if st.get('sigma'):
        sm[pos] -= st['sigma'] * mass


def prepare(case, seed):
    kind = case['kind']
    if kind == 'batch':
        ns, sigma, loads = _batch_draws(case, seed)
        systems = []
        for n, sg, b in zip(ns, sigma, loads):
            hs = _system(n)
            systems.append(dict(hs=hs, sm=system.shift_diagonal(_unit_sm(n), *_mass(n), sg), b=b.T))
        return dict(kind=kind, solver=batch.BatchSolver(systems))
    n = case['n']
    hs = _system(n)
    if kind == 'assemble':
        g = np.random.default_rng([seed, 4])
        xyz = hs.box.node_coords() + g.uniform(-case['amp'], case['amp'], size=(hs.box.nanod, 3))
        moduli = g.uniform(0.1, 1.0, size=hs.box.nel)
        return dict(kind=kind, elements=_elements(n), xyz=torch.from_numpy(xyz).cuda(),
                    moduli=torch.from_numpy(moduli).cuda(),
                    em=torch.empty((hs.box.nel, 24, 24), dtype=torch.float64, device='cuda'),
                    sm=torch.empty(hs.neq + hs.nzerol, dtype=torch.float64, device='cuda'))
    if kind == 'adjoint':
        g = np.random.default_rng([seed, 5])
        shape = (hs.neq,) if case['nrhs'] == 1 else (case['nrhs'], hs.neq)
        theta = torch.from_numpy(g.uniform(0.2, 1.0, size=hs.box.nel)).cuda()
        f = torch.from_numpy(g.uniform(-1.0, 1.0, size=shape)).cuda()
        gu = torch.from_numpy(g.uniform(-1.0, 1.0, size=shape)).cuda()
        return dict(kind=kind, model=adjoint.SimpModel(hs), theta=theta, f=f, gu=gu)
    st = dict(kind=kind, n=n, nrhs=case['nrhs'], sigma=_sigma(case))
    st['moduli'] = torch.from_numpy(_moduli(case, seed)).cuda()
    loads = torch.from_numpy(_loads(case, seed))
    sm = torch.empty(hs.neq + hs.nzerol, dtype=torch.float64, device='cuda')
    if kind == 'sprsol':
        _assembled(st, sm)
        st['sm0'] = sm.cpu()
        st['sm'] = torch.empty_like(st['sm0']).pin_memory()
        st['b0'] = loads
        st['b'] = torch.empty_like(loads).pin_memory()
        st['mspar'], st['mspar0'] = hs.mspar, hs.mspar.copy()
        st['mtrees'], st['msifa'] = hs.mtrees, hs.msifa
        return st
    st.update(sm=sm, b0=loads.cuda(), solver=spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa),
              stream=torch.cuda.Stream())
    st['solver'].set_stream(st['stream'].cuda_stream)
    st['b'] = torch.empty_like(st['b0'])
    if kind == 'factor_solve':
        st['rule'] = case['rule']
        if st['rule'] == 'replace':
            st['dcor'] = torch.empty(2 * hs.neq, dtype=torch.float64, device='cuda')
    elif kind == 'mixed':
        st['solver'].set_mode(1)
    else:
        st['sweeps'] = case['sweeps']
        _assembled(st, sm)
        torch.cuda.synchronize()
        st['solver'].factor(sm)
    torch.cuda.synchronize()
    return st


# ---- one pass

def run(st):
    kind = st['kind']
    if kind == 'batch':
        bs = st['solver']
        r = bs.run()
        return dict(sm=bs.sm, x=bs.b, numneg=bs.numneg(), tol2=r['tol2'])
    if kind == 'adjoint':
        theta = st['theta'].detach().requires_grad_(True)
        f = st['f'].detach().requires_grad_(True)
        u = adjoint.simp_solve(theta, f, st['model'])
        u.backward(st['gu'])
        return dict(u=u.detach(), theta=theta.grad, f=f.grad)
    if kind == 'assemble':
        st['elements'].hex8(st['xyz'], st['moduli'], out=st['em'])
        st['elements'].assemble(st['sm'], st['em'])
        return dict(em=st['em'], sm=st['sm'])
    if kind == 'sprsol':
        st['sm'].copy_(st['sm0'])
        st['b'].copy_(st['b0'])
        st['mspar'][:] = st['mspar0']
        tol = np.array([1e-12, 0.0, 0.0])
        b = st['b'].numpy().T
        ierr = spr.sprsol(3, st['mspar'], st['mtrees'], st['msifa'], st['sm'].numpy(), b, b.shape[0], st['nrhs'], tol)
        return dict(sm=st['sm'], x=st['b'], ierr=ierr, numneg=int(st['mspar'][25]), tol=tol[1:])
    ds, sm, b, nrhs = st['solver'], st['sm'], st['b'], st['nrhs']
    with torch.cuda.stream(st['stream']):
        if kind == 'solve':
            b.copy_(st['b0'])
            if st['sweeps'] == 'split':
                ds.solve(sm, b, nrhs, which=1)
                ds.solve(sm, b, nrhs, which=2)
            else:
                ds.solve(sm, b, nrhs, which={'both': 3, 'forward': 1, 'back': 2}[st['sweeps']])
            return dict(x=b)
        _assembled(st, sm)
        if kind == 'mixed':
            ds.build_residual(sm)
            r = ds.factor(sm)
            ds.refine(sm, st['b0'], b, nrhs, tol=1e-13)
            return dict(x=b, numneg=r['numneg'])
        b.copy_(st['b0'])
        if st['rule'] == 'replace':
            r = ds.factor3(sm, st['dcor'])
        else:
            r = ds.factor(sm)
        ds.solve(sm, b, nrhs)
        out = dict(sm=sm, x=b, numneg=r['numneg'], lierr=r['lierr'], tol2=r['tol2'], tol3=r['tol3'])
        if st['rule'] == 'replace':
            out['dcor'] = st['dcor']
        return out


# ---- the work a pass cannot do without

def work(case):
    kind = case['kind']
    if kind == 'batch':
        hs = [_system(n) for n in _batch_sizes(case)]
        return dict(bytes=sum(16.0 * (h.neq + h.nzerol) + 16.0 * h.neq * case['nrhs'] for h in hs),
                    flops=sum(float(h.rinfo[2]) + case['nrhs'] * float(h.rinfo[3]) for h in hs))
    hs = _system(case['n'])
    sm, nel = 8.0 * (hs.neq + hs.nzerol), hs.box.nel
    if kind == 'assemble':
        # coordinates and moduli in, element matrices out and in again, SM out
        return dict(bytes=24.0 * hs.box.nanod + 8.0 * nel + 2 * 8.0 * 576 * nel + sm, flops=nel * (8 * 64 * 45 + 576.0))
    vec, sweeps = 8.0 * hs.neq * case['nrhs'], float(hs.rinfo[3]) * case['nrhs']
    if kind == 'solve':
        reads = 2 if case['sweeps'] == 'split' else 1
        half = 0.5 if case['sweeps'] in ('forward', 'back') else 1.0
        return dict(bytes=reads * (sm + 2 * vec), flops=half * sweeps)
    if kind == 'adjoint':
        return dict(bytes=sm + 4 * vec + 16.0 * nel, flops=float(hs.rinfo[2]) + 2 * sweeps)
    if kind == 'sprsol':
        return dict(bytes=2 * sm + 2 * vec, flops=float(hs.rinfo[2]) + sweeps)
    return dict(bytes=8.0 * nel + sm + 2 * vec, flops=float(hs.rinfo[2]) + sweeps)


# ---- the same results from plain 64-bit torch

def _cg(apply, diag, b, most=20000):
    """Conjugate gradients with diagonal scaling, all right-hand sides at once, to the limit of FP64."""
    x = torch.zeros_like(b)
    for _ in range(3):                               # restarted on the true residual
        r = b - apply(x)
        z = r / diag
        p, rz, first = z, (r * z).sum(1), (b * b / diag).sum(1)
        for it in range(most):
            q = apply(p)
            a = rz / (p * q).sum(1)
            x = x + a[:, None] * p
            r = r - a[:, None] * q
            z = r / diag
            new = (r * z).sum(1)
            if it % 25 == 24 and bool((new <= 1e-32 * first).all()):
                break
            p = z + (new / rz)[:, None] * p
            rz = new
    return x


class _Matrix:
    """K = sum_e E_e K_ref - sigma M, applied element by element or made dense."""

    def __init__(self, n, moduli, sigma=0.0):
        hs = _system(n)
        self.neq, self.sigma = hs.neq, sigma
        eq = torch.from_numpy(hs.element_equations()).cuda()
        self.eq = torch.where(eq < 0, self.neq, eq)              # a spare last row takes the clamped DOFs
        self.ke = torch.from_numpy(np.ascontiguousarray(hs.ke)).cuda()
        self.e = torch.as_tensor(moduli, dtype=torch.float64).cuda()
        self.mass = torch.from_numpy(hs.to_internal(hs.box.lumped_mass())).cuda()

    def apply(self, x):
        xe = torch.nn.functional.pad(x, (0, 1))[:, self.eq]
        y = torch.zeros((x.shape[0], self.neq + 1), dtype=torch.float64, device='cuda')
        y.index_add_(1, self.eq.reshape(-1), ((xe @ self.ke) * self.e[:, None]).reshape(x.shape[0], -1))
        return y[:, :-1] - self.sigma * self.mass * x

    def diag(self):
        d = torch.zeros(self.neq + 1, dtype=torch.float64, device='cuda')
        d.index_add_(0, self.eq.reshape(-1), (self.ke.diagonal() * self.e[:, None]).reshape(-1))
        return d[:-1] - self.sigma * self.mass

    def dense(self):
        m = self.neq + 1
        k = torch.zeros(m * m, dtype=torch.float64, device='cuda')
        at = self.eq[:, :, None] * m + self.eq[:, None, :]
        k.index_add_(0, at.reshape(-1), (self.ke * self.e[:, None, None]).reshape(-1))
        k = k.view(m, m)[:-1, :-1].clone()
        k.diagonal().sub_(self.sigma * self.mass)
        return k

    def solve(self, b):
        if self.neq <= 15000:
            return torch.linalg.solve(self.dense(), b.T).T
        return _cg(self.apply, self.diag(), b)


def _packed(n, low):
    """SM's LNZ layout (column j of a supernode: its rows j, j + 1, ...) of a dense lower triangle."""
    hs = _system(n)
    m, ns = hs.mspar, int(hs.mspar[10])
    xs, xl = hs.mtrees[m[44] - 1: m[44] + ns], hs.mtrees[m[45] - 1: m[45] + ns]
    lindx = hs.msifa[m[46] - 1:]
    rows, cols = [], []
    for s in range(ns):
        r = lindx[xl[s] - 1: xl[s + 1] - 1] - 1
        for j in range(int(xs[s + 1] - xs[s])):
            rows.append(r[j:])
            cols.append(np.full(len(r) - j, xs[s] - 1 + j))
    return low[torch.from_numpy(np.concatenate(rows)).cuda(), torch.from_numpy(np.concatenate(cols)).cuda()]


def _exact_hex8(xyz, moduli, conn, nu=0.3):
    """Element matrices (nel, 24, 24): sum over the 2x2x2 Gauss points of det J B' D B."""
    corners = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                            [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64)
    xe = torch.from_numpy(xyz)[torch.from_numpy(conn - 1)]
    mu = torch.from_numpy(moduli / (2 * (1 + nu)))[:, None, None, None, None]
    lam = torch.from_numpy(moduli * nu / ((1 + nu) * (1 - 2 * nu)))[:, None, None, None, None]
    k = torch.zeros((len(conn), 8, 3, 8, 3), dtype=torch.float64)
    eye = torch.eye(3, dtype=torch.float64)
    for gp in corners / math.sqrt(3.0):
        t = 1 + gp * corners
        dn = corners * torch.stack([t[:, 1] * t[:, 2], t[:, 0] * t[:, 2], t[:, 0] * t[:, 1]], 1) / 8
        jac = torch.einsum('ai,eaj->eij', dn, xe)
        g = torch.linalg.solve(jac, dn.T.expand(len(conn), 3, 8)).transpose(1, 2)
        gg = torch.einsum('eai,ebj->eaibj', g, g)
        dot = torch.einsum('eai,ebi->eab', g, g)[:, :, None, :, None] * eye[:, None, :]
        k += torch.linalg.det(jac)[:, None, None, None, None] * (lam * gg + mu * (gg.transpose(2, 4) + dot))
    return k.reshape(len(conn), 24, 24)


def exact(case, seed):
    kind = case['kind']
    if kind == 'batch':
        ns, sigma, loads = _batch_draws(case, seed)
        x = [_Matrix(n, np.ones(n ** 3), sg).solve(torch.from_numpy(b).cuda()) for n, sg, b in zip(ns, sigma, loads)]
        return dict(sm=None, x=torch.cat(x, 1), numneg=None, tol2=None)
    if kind == 'assemble':
        st = prepare(case, seed)
        em = _exact_hex8(st['xyz'].cpu().numpy(), st['moduli'].cpu().numpy(), _system(case['n']).box.conn)
        return dict(em=em, sm=None)
    if kind == 'adjoint':
        st = prepare(case, seed)
        theta, f, gu = st['theta'], st['f'].reshape(-1, st['f'].shape[-1]), st['gu'].reshape(-1, st['gu'].shape[-1])
        m = _Matrix(case['n'], (theta ** 3).cpu())
        u, lam = m.solve(f), m.solve(gu)
        ue, le = (torch.nn.functional.pad(v, (0, 1))[:, m.eq] for v in (u, lam))
        grad = -3 * theta ** 2 * ((ue @ m.ke) * le).sum((0, 2))
        return dict(u=u.reshape(st['f'].shape), theta=grad, f=lam.reshape(st['f'].shape))
    if case['n'] > 32 or (_sigma(case) and case['n'] > 16) or case.get('sweeps') in ('forward', 'back'):
        return None
    m = _Matrix(case['n'], _moduli(case, seed), _sigma(case))
    x = m.solve(torch.from_numpy(_loads(case, seed)).cuda())
    if kind in ('mixed', 'solve'):
        return dict(x=x)
    sm = None
    if case['n'] <= 12 and not _sigma(case):
        c = torch.linalg.cholesky(m.dense())
        d = c.diagonal() ** 2
        low = c / c.diagonal()
        low.diagonal().copy_(d)
        sm = torch.cat([d, _packed(case['n'], low)])
    return dict(sm=sm, x=x)
