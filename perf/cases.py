"""The calls whose speed matters to a user of bolt_b200, and their answers in
plain 64-bit torch.

``listed()`` names twelve of them, ``draw(rng)`` makes more of the same kinds.
``prepare`` builds what a program holds before its time loop (a solver, a
batch, a rollout), ``run`` is one pass of that loop through the public entry
points, ``exact`` restates the pass without the package.
"""

import math
import types

import torch

from bolt_b200.adjoint import Rollout1D1V, rollout
from bolt_b200.batch import BatchSolver
from bolt_b200.nonlinear_solver import nonlinear_solver
from bolt_b200.physical_system import physical_system
import bolt_b200.src.nonrelativistic_boltzmann.advection_terms as advection
import bolt_b200.src.nonrelativistic_boltzmann.collision_operator as collision
import bolt_b200.src.nonrelativistic_boltzmann.moments as moments

NG = 3
TAU = 0.05


def _fvm(name, precision, q, p, recon='weno5', bc='periodic', integrator='RK4', source=True,
         fields='none', species=1, method='FVM'):
    return dict(name=name, path='solver', precision=precision, N_q1=q[0], N_q2=q[1], N_p1=p[0],
                N_p2=p[1], N_p3=p[2], recon=recon, bc=bc, integrator=integrator, source=source,
                fields=fields, species=species, method=method)


def listed():
    return [
        # relaxation run at the size of a first test script: launches and host time count
        _fvm('relax 1D1V fp64', 'fp64', (64, 1), (128, 1, 1), integrator='RK2'),
        # Landau damping: the Poisson solve at every df/dt
        _fvm('landau 1D1V fp64', 'fp64', (128, 1), (256, 1, 1), integrator='RK2', source=False,
             fields='electrostatic'),
        # collisionless plasma on Yee-grid fields, both precisions that such runs use
        _fvm('fdtd 2D2V fp64', 'fp64', (64, 64), (32, 32, 1), source=False,
             fields='electrodynamic'),
        _fvm('fdtd 2D2V fp32', 'fp32', (64, 64), (32, 32, 1), source=False,
             fields='electrodynamic'),
        # the reference's own performance script: 32^2 x 20^3, minmod, fields, RK2
        _fvm('fdtd minmod 2D3V fp32', 'fp32', (32, 32), (20, 20, 20), recon='minmod',
             integrator='RK2', source=False, fields='electrodynamic'),
        # walls, and sizes that no tile divides
        _fvm('mirror 2D2V odd fp32', 'fp32', (75, 50), (45, 35, 1), bc='mirror',
             integrator='RK2'),
        # the default precision in 2D3V
        _fvm('bgk 2D3V fp64', 'fp64', (64, 64), (24, 24, 24)),
        # production size: single precision, and the FP64 throughput form
        _fvm('bgk 2D3V fp32', 'fp32', (128, 128), (24, 24, 24)),
        _fvm('bgk 2D3V fp64-fast', 'fp64-fast', (128, 128), (24, 24, 24)),
        # semi-Lagrangian in q, Strang splitting
        _fvm('semi-lagrangian 2D3V fp32', 'fp32', (128, 128), (24, 24, 24), method='ASL'),
        # a parameter sweep of 256 ragged 1D1V runs
        dict(name='batch of 256 runs', path='batch', runs=256, sweep=0, steps=5),
        # gradient of a rollout: forward and backward
        dict(name='adjoint 1D1V fp32', path='adjoint', precision='fp32', N_q1=128, N_p1=256,
             steps=100, snapshots=10),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['1d1v', '2d2v', '2d2v', '2d3v', '2d3v', 'asl', 'batch', 'adjoint'])
    if kind == 'batch':
        return dict(path='batch', runs=_between(rng, 8, 256), sweep=rng.randrange(1, 1000),
                    steps=rng.randrange(1, 6))
    if kind == 'adjoint':
        return dict(path='adjoint', precision=rng.choice(['fp32', 'fp64']),
                    N_q1=_between(rng, 24, 160), N_p1=_between(rng, 32, 320),
                    steps=rng.randrange(20, 101), snapshots=rng.randrange(4, 11))
    precision = rng.choice(['fp64', 'fp32', 'fp64-fast'])
    integrator = rng.choice(['RK2', 'RK4'])
    recon = rng.choice(['weno5', 'weno5', 'minmod', 'ppm'])
    if kind == '1d1v':
        c = _fvm('', precision, (_between(rng, 16, 512), 1), (_between(rng, 32, 1024), 1, 1),
                 recon=recon, integrator=integrator)
        if rng.random() < 0.4:
            c.update(fields='electrostatic', source=False)
    elif kind == '2d2v':
        # (p grids that resolve the distribution: cells of up to one thermal speed)
        species = rng.choice([1, 1, 2])
        lo = 20 if species == 1 else 28
        c = _fvm('', precision, (_between(rng, 8, 140), _between(rng, 8, 140)),
                 (_between(rng, lo, 48), _between(rng, lo, 48), 1), recon=recon,
                 integrator=integrator, species=species)
        if rng.random() < 0.5:
            c.update(fields='electrodynamic', source=False)
        elif rng.random() < 0.5:
            c.update(bc='mirror')
    else:
        top = 72 if precision == 'fp64' else 112
        q = (_between(rng, 8, top), _between(rng, 8, top))
        if rng.random() < 0.5:                    # whole tiles, as production runs choose
            q = tuple(max(8, n // 8 * 8) for n in q)
        n = _between(rng, 14, 24)
        p = (max(16, n // 8 * 8),) * 3 if rng.random() < 0.5 else (n, _between(rng, 14, 24), n)
        c = _fvm('', precision, q, p, recon=recon, integrator=integrator,
                 source=kind == 'asl' or rng.random() < 0.8)
        if kind == 'asl':
            c.update(method='ASL', recon='weno5', integrator='RK4')
            if precision == 'fp64-fast':
                c['precision'] = 'fp64'
        elif rng.random() < 0.3:
            c.update(bc='mirror')
    del c['name']
    return c


# ---------------------------------------------------------------------------------------------
# the problem of a case, in plain numbers
# ---------------------------------------------------------------------------------------------
class _Problem(object):
    """Grid, physics and initial state of a solver case: density waves with a
    little cell-to-cell noise times drifting Maxwellians."""

    def __init__(self, c, seed):
        g = torch.Generator().manual_seed(int(seed))
        u = lambda lo, hi: lo + (hi - lo) * float(torch.rand((), generator=g, dtype=torch.float64))
        self.c = c
        self.N = (c['N_q1'], c['N_q2'])
        self.P = (c['N_p1'], c['N_p2'], c['N_p3'])
        self.p_dim = 1 if self.P[1] == 1 else (2 if self.P[2] == 1 else 3)
        self.p_max = {1: 10.0, 2: 8.0, 3: 6.0}[self.p_dim]
        self.species = c['species']
        self.mass = [1.0, 2.0][:self.species]
        self.charge = ([-1.0, 1.0] if c['fields'] != 'none' else [0.0, 0.0])[:self.species]
        self.dq = [1.0 / n for n in self.N]
        lim = [0.5 if n == 1 else self.p_max for n in self.P]
        self.p_lim = lim
        self.dp = [2 * h / n for h, n in zip(lim, self.P)]
        cfl = 1.7 if c['method'] == 'ASL' else 0.15
        self.dt = cfl * min(self.dq[d] for d in range(2) if self.N[d] > 1) / self.p_max
        self.T = u(0.9, 1.1)
        self.drift = [u(-0.2, 0.2) for _ in range(3)]
        self.amp, self.phase = u(0.05, 0.1), (u(0, 6.28), u(0, 6.28))
        self.noise = 1e-3 * torch.randn(self.N[0], self.N[1], generator=g, dtype=torch.float64)

    def density(self, q1, q2):
        """At cell centres (any shape; ghost centres wrap around)."""
        n = 1 + self.amp * torch.cos(2 * math.pi * q1 + self.phase[0])
        if self.N[1] > 1:
            n = n * (1 + self.amp * torch.cos(2 * math.pi * q2 + self.phase[1]))
        i = torch.floor(q1 / self.dq[0]).long() % self.N[0]
        j = torch.floor(q2 / self.dq[1]).long() % self.N[1]
        return n * (1 + self.noise.to(n.device)[i, j])

    def f0(self, q1, q2, p, mass):
        f = self.density(q1, q2)
        for d in range(self.p_dim):
            f = f * torch.sqrt(mass / (2 * math.pi * self.T)) \
                * torch.exp(-mass * (p[d] - self.drift[d]) ** 2 / (2 * self.T))
        return f

    def system(self):
        c = self.c
        dom = types.ModuleType('domain')
        dom.N_q1, dom.N_q2 = self.N
        dom.N_p1, dom.N_p2, dom.N_p3 = self.P
        dom.N_ghost = NG
        dom.q1_start = dom.q2_start = 0.0
        dom.q1_end = dom.q2_end = 1.0
        for d in range(3):
            setattr(dom, 'p%d_start' % (d + 1), [-self.p_lim[d]] * self.species)
            setattr(dom, 'p%d_end' % (d + 1), [self.p_lim[d]] * self.species)
        bc = types.ModuleType('boundary_conditions')
        bc.in_q1_left = bc.in_q1_right = c['bc']
        bc.in_q2_bottom = bc.in_q2_top = c['bc']
        es = c['fields'] == 'electrostatic'
        params = types.ModuleType('params')
        for k, v in dict(
                fields_enabled=c['fields'] != 'none',
                fields_type='electrostatic' if es else 'electrodynamic',
                fields_initialize='fft', fields_solver='fft' if es else 'fdtd',
                solver_method_in_q=c['method'], solver_method_in_p='FVM',
                reconstruction_method_in_q=c['recon'], reconstruction_method_in_p=c['recon'],
                riemann_solver_in_q='upwind-flux', riemann_solver_in_p='upwind-flux',
                p_dim=self.p_dim, num_devices=1, mass=list(self.mass),
                charge=list(self.charge), boltzmann_constant=1.0, source_enabled=c['source'],
                instantaneous_collisions=False, hybrid_model_enabled=False, eps=1.0, mu=1.0,
                p_space_grid='cartesian', time_integrator=c['integrator'],
                precision=c['precision']).items():
            setattr(params, k, v)
        params.tau = lambda q1, q2, p1, p2, p3: TAU * p1 ** 0 * q1 ** 0
        ini = types.ModuleType('initialize')
        ini.initialize_f = lambda q1, q2, p1, p2, p3, params: \
            self.f0(q1, q2, (p1, p2, p3), params.mass)
        return physical_system(dom, bc, params, ini, advection, collision.BGK, moments)


class _Sweep(object):
    """The runs of a batch case: grid sizes from the sweep's number, collision
    times, amplitudes and wavenumbers from the seed."""

    def __init__(self, c, seed):
        g = torch.Generator().manual_seed(1000 + c['sweep'])
        h = torch.Generator().manual_seed(int(seed))
        pick = lambda gen, n: int(torch.randint(n, (), generator=gen))
        frac = lambda: float(torch.rand((), generator=h, dtype=torch.float64))
        self.runs = []
        for _ in range(c['runs']):
            nq, npp = 32 + 16 * pick(g, 15), 64 + 32 * pick(g, 15)
            self.runs.append(dict(N_q1=nq, N_p1=npp, tau=10 ** (-3 + 2 * frac()),
                                  amp=10 ** (-3 + 2 * frac()), k=1 + pick(h, 4),
                                  dt=0.5 / nq / 10.0))

    @staticmethod
    def f0(run, q1, p1):
        return (1 + run['amp'] * torch.cos(2 * math.pi * run['k'] * q1)) \
            * math.sqrt(1 / (2 * math.pi)) * torch.exp(-p1 ** 2 / 2)

    def system(self, run):
        dom = types.ModuleType('domain')
        dom.N_q1, dom.N_p1 = run['N_q1'], run['N_p1']
        dom.N_q2 = dom.N_p2 = dom.N_p3 = 1
        dom.N_ghost = NG
        dom.q1_start = dom.q2_start = 0.0
        dom.q1_end = dom.q2_end = 1.0
        dom.p1_start, dom.p1_end = [-10.0], [10.0]
        dom.p2_start, dom.p2_end, dom.p3_start, dom.p3_end = [-0.5], [0.5], [-0.5], [0.5]
        bc = types.ModuleType('boundary_conditions')
        bc.in_q1_left = bc.in_q1_right = bc.in_q2_bottom = bc.in_q2_top = 'periodic'
        params = types.ModuleType('params')
        for k, v in dict(fields_enabled=False, fields_type='electrodynamic',
                         fields_initialize='fft', fields_solver='fdtd',
                         solver_method_in_q='FVM', solver_method_in_p='FVM',
                         reconstruction_method_in_q='weno5', reconstruction_method_in_p='weno5',
                         riemann_solver_in_q='upwind-flux', riemann_solver_in_p='upwind-flux',
                         p_dim=1, num_devices=1, mass=[1.0], charge=[0.0],
                         boltzmann_constant=1.0, source_enabled=True,
                         instantaneous_collisions=False, hybrid_model_enabled=False, eps=1.0,
                         mu=1.0, p_space_grid='cartesian', time_integrator='RK4',
                         precision='fp32').items():
            setattr(params, k, v)
        params.tau = lambda q1, q2, p1, p2, p3: run['tau'] * p1 ** 0 * q1 ** 0
        ini = types.ModuleType('initialize')
        ini.initialize_f = lambda q1, q2, p1, p2, p3, params: self.f0(run, q1, p1)
        return physical_system(dom, bc, params, ini, advection, collision.BGK, moments)


def _rollout_inputs(c, seed):
    """f0 (N_q1, N_p1), tau and dt of an adjoint case: a perturbed Maxwellian."""
    g = torch.Generator().manual_seed(int(seed))
    amp, tau, phase = (float(x) for x in torch.rand(3, generator=g, dtype=torch.float64))
    q = (torch.arange(c['N_q1'], dtype=torch.float64) + 0.5) / c['N_q1']
    p = -6.0 + (torch.arange(c['N_p1'], dtype=torch.float64) + 0.5) * 12.0 / c['N_p1']
    n = 1 + (0.05 + 0.1 * amp) * torch.cos(2 * math.pi * (q + phase))
    f0 = n[:, None] * torch.exp(-p ** 2 / 2)[None] / math.sqrt(2 * math.pi)
    return f0, 0.05 + 0.05 * tau, 0.2 / c['N_q1'] / 6.0


# ---------------------------------------------------------------------------------------------
# the pass
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    if c['path'] == 'batch':
        s = _Sweep(c, seed)
        batch = BatchSolver([s.system(r) for r in s.runs], [r['dt'] for r in s.runs])
        # all runs' f as one tensor: whole multiples of 128 bytes, packed end to end
        cells = sum((r['N_q1'] + 2 * NG) * r['N_p1'] for r in s.runs)
        f = batch.f(0).as_strided((cells,), (1,), batch.f(0).storage_offset())
        f.batch = batch           # the batch owns the memory: alive as long as its f
        return dict(case=c, batch=batch, f=f)
    if c['path'] == 'adjoint':
        f0, tau, dt = _rollout_inputs(c, seed)
        roll = Rollout1D1V(N_q1=c['N_q1'], N_p1=c['N_p1'], p1_start=-6.0, p1_end=6.0, dt=dt,
                           tau=tau, nsteps=c['steps'], snapshots=c['snapshots'],
                           precision=c['precision'])
        return dict(case=c, roll=roll, f0=f0.cuda().requires_grad_(),
                    tau=torch.tensor(tau, dtype=torch.float64, requires_grad=True))
    pr = _Problem(c, seed)
    return dict(case=c, dt=pr.dt, solver=nonlinear_solver(pr.system()))


def run(state):
    c = state['case']
    if c['path'] == 'batch':
        state['batch'].run(c['steps'])
        return state['f']
    if c['path'] == 'adjoint':
        f0, tau = state['f0'], state['tau']
        f0.grad = tau.grad = None
        J = rollout(f0, tau, state['roll'])
        J.backward()
        return dict(J=J.detach(), f0=f0.grad, tau=tau.grad)
    nls = state['solver']
    nls.strang_timestep(state['dt'])
    inner = slice(NG, -NG)
    out = dict(f=nls.f[:, :, inner, inner])
    # the diagnostics a script records each step: the density of small runs,
    # the fields where there are any
    if c['N_q2'] == 1:
        out['density'] = nls.compute_moments('density')[:, :, inner, inner]
    if c['fields'] == 'electrodynamic':
        out['fields'] = nls.fields_solver.yee_grid_EM_fields[:, :, inner, inner]
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
# operations of one face value (WENO5: a new smoothness indicator, its weight
# and the weighted sum, neighbours' shared; minmod, PPM: the limiter)
FACE_OPS = {'weno5': 18, 'minmod': 10, 'ppm': 40}


def _words(integrator):
    # f read and written once per stage, with the bases and accumulators of the
    # scheme: 5 words per RK2 step, 17 per classic RK4 step
    return 5 if integrator == 'RK2' else 17


def work(case):
    c = case
    if c['path'] == 'batch':
        runs = _Sweep(c, 0).runs
        cells = sum(r['N_q1'] * r['N_p1'] for r in runs) * c['steps']
        return dict(bytes=cells * 17 * 4, flops=cells * 4 * (2 * FACE_OPS['weno5'] + 12))
    if c['path'] == 'adjoint':
        cells = c['N_q1'] * c['N_p1'] * c['steps']
        word = 4 if c['precision'] == 'fp32' else 8
        # forward, forward again, backward at about twice a forward
        return dict(bytes=cells * 4 * 17 * word, flops=cells * 4 * 4 * (2 * FACE_OPS['weno5'] + 12))
    cells = c['N_q1'] * c['N_q2'] * c['N_p1'] * c['N_p2'] * c['N_p3'] * c['species']
    word = 4 if c['precision'] == 'fp32' else 8
    if c['method'] == 'ASL':
        # two interpolations (read, write) and the two stages of the source
        return dict(bytes=cells * 8 * word, flops=cells * (2 * 40 + 2 * 12))
    stages = 2 if c['integrator'] == 'RK2' else 4
    axes = sum(n > 1 for n in (c['N_q1'], c['N_q2']))
    if c['fields'] != 'none':
        axes += sum(n > 1 for n in (c['N_p1'], c['N_p2'], c['N_p3']))
    per_cell = axes * (2 * FACE_OPS[c['recon']] + 3) + (8 if c['source'] else 0) + 12
    return dict(bytes=cells * _words(c['integrator']) * word, flops=cells * stages * per_cell)


def tolerance(case):
    # about four times the distance from exact() over the ranges; the adjoint's
    # is set by the gradient in tau, a sum with cancellation
    if case['path'] == 'adjoint':
        return dict(rel=1e-3 if case['precision'] == 'fp32' else 1e-10, max=0.05)
    if case['path'] == 'batch':
        return dict(rel=1e-6)
    return dict(rel=5e-7 if case['precision'] == 'fp32' else 4e-13)


# ---------------------------------------------------------------------------------------------
# the same pass in plain FP64 torch: arrays (q2, q1, species, p3, p2, p1), interior cells only
# ---------------------------------------------------------------------------------------------
Q2, Q1, P3, P2, P1 = 0, 1, 3, 4, 5


def _weno5(y, right):
    def beta(a, b, c):
        return (4 / 3 * a * a - 19 / 3 * a * b + 25 / 3 * b * b + 11 / 3 * a * c
                - 31 / 3 * b * c + 10 / 3 * c * c) + 1e-17 * (1 + a.abs() + b.abs() + c.abs())
    y0, y1, y2, y3, y4 = y
    if not right:
        # the left face is the right face of the mirrored window; the first
        # indicator's polynomial is not symmetric, so the weights are spelled out
        u = (-0.125 * y0 + 0.75 * y1 + 0.375 * y2, 0.375 * y1 + 0.75 * y2 - 0.125 * y3,
             1.875 * y2 - 1.25 * y3 + 0.375 * y4)
        g = (5 / 16, 5 / 8, 1 / 16)
    else:
        u = (0.375 * y0 - 1.25 * y1 + 1.875 * y2, -0.125 * y1 + 0.75 * y2 + 0.375 * y3,
             0.375 * y2 + 0.75 * y3 - 0.125 * y4)
        g = (1 / 16, 5 / 8, 5 / 16)
    num = den = 0.0
    for k, s in enumerate(((y0, y1, y2), (y1, y2, y3), (y2, y3, y4))):
        w = g[k] / beta(*s) ** 2
        num, den = num + w * u[k], den + w
    return num / den


def _minmod(y, right):
    y2 = y[2]
    a, b, c = 2 * (y2 - y[1]), 0.5 * (y[3] - y[1]), 2 * (y[3] - y2)
    m = torch.minimum(torch.minimum(a.abs(), b.abs()), c.abs())
    same = ((a < 0) == (b < 0)) & ((a < 0) == (c < 0))
    s = torch.where(same, torch.where(a < 0, -m, m), torch.zeros_like(m))
    return y2 + 0.5 * s if right else y2 - 0.5 * s


def _ppm(y, right):
    y0, y1, y2, y3, y4 = y

    def slope(a, b, c):
        d, lo, hi = 0.5 * (c - a), 2 * (b - a), 2 * (c - b)
        m = torch.minimum(d.abs(), torch.minimum(lo.abs(), hi.abs()))
        return torch.where(lo * hi <= 0, torch.zeros_like(m), torch.where(d > 0, m, -m))
    s1, s2, s3 = slope(y0, y1, y2), slope(y1, y2, y3), slope(y2, y3, y4)
    left = 0.5 * (y2 + y1) - (s2 - s1) / 6
    rite = 0.5 * (y3 + y2) - (s3 - s2) / 6
    flat = (rite - y2) * (y2 - left) <= 0
    d = rite - left
    e = 6 * (y2 - 0.5 * (rite + left))
    c2, c3 = d * (d - e) < 0, d * (d + e) < 0
    left, rite = torch.where(flat, y2, left), torch.where(flat, y2, rite)
    left = torch.where(c2, 3 * y2 - 2 * rite, left)
    rite = torch.where(c2, rite, torch.where(c3, 3 * y2 - 2 * left, rite))
    return rite if right else left


FACES = dict(weno5=_weno5, minmod=_minmod, ppm=_ppm)


def _padded(f, axis, mirror):
    """Three more cells on each side of an axis: around the period, or the
    mirror image with the normal velocity reversed."""
    n = f.shape[axis]
    if not mirror:
        i = torch.arange(-NG, n + NG, device=f.device) % n
        return f.index_select(axis, i)
    lo, hi = f.narrow(axis, 0, NG).flip(axis), f.narrow(axis, n - NG, NG).flip(axis)
    v = P1 if axis == Q1 else P2
    return torch.cat([lo.flip(v), f, hi.flip(v)], axis)


def _left_faces(f, axis, speed, recon, mirror=False):
    """Upwind value at the left face of every cell, and of the cell past the
    last, along an axis; `speed` broadcasts against f and is constant along it."""
    n = f.shape[axis]
    g = _padded(f, axis, mirror)
    # face i lies between padded cells i + 2 and i + 3
    win = lambda first: [g.narrow(axis, first + t, n + 1) for t in range(5)]
    face = FACES[recon]
    return torch.where(speed > 0, face(win(0), True), face(win(1), False))


def _difference(F, axis):
    n = F.shape[axis] - 1
    return F.narrow(axis, 1, n) - F.narrow(axis, 0, n)


class _Exact(object):

    def __init__(self, c, seed):
        self.pr = pr = _Problem(c, seed)
        self.c = c
        dev = 'cuda' if torch.cuda.is_available() else 'cpu'
        centre = lambda n, d, lo: lo + (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) * d
        q1 = centre(pr.N[0], pr.dq[0], 0.0).reshape(1, -1, 1, 1, 1, 1)
        q2 = centre(pr.N[1], pr.dq[1], 0.0).reshape(-1, 1, 1, 1, 1, 1)
        self.v = [centre(pr.P[d], pr.dp[d], -pr.p_lim[d]).reshape(
            [1, 1, 1] + [pr.P[d] if a == d else 1 for a in (2, 1, 0)]) for d in range(3)]
        per = lambda x: torch.tensor(x, dtype=torch.float64, device=dev).reshape(1, 1, -1, 1, 1, 1)
        self.mass, self.charge = per(pr.mass), per(pr.charge)
        self.f = pr.f0(q1, q2, self.v, self.mass)
        self.measure = pr.dp[0] * pr.dp[1] * pr.dp[2]
        self.mirror = c['bc'] == 'mirror'
        if c['fields'] != 'none':
            zero = torch.zeros(pr.N[1], pr.N[0], dtype=torch.float64, device=dev)
            self.cell = self._poisson(self.f) + [zero] * 4
            E1, E2 = self.cell[:2]
            self.yee = [0.5 * (E1 + E1.roll(1, 1)), 0.5 * (E2 + E2.roll(1, 0))] + [zero] * 4

    # moments: (q2, q1, species, 1, 1, 1)
    def _moment(self, f):
        return f.sum((P3, P2, P1), keepdim=True) * self.measure

    def _charge_sum(self, f):
        return (self.charge * self._moment(f)).sum(2)[:, :, 0, 0, 0]

    def _poisson(self, f):
        rho = self._charge_sum(f)
        k1 = torch.fft.fftfreq(self.pr.N[0], self.pr.dq[0], dtype=torch.float64).to(rho.device)
        k2 = torch.fft.fftfreq(self.pr.N[1], self.pr.dq[1], dtype=torch.float64).to(rho.device)
        k1, k2 = k1[None, :], k2[:, None]
        ksq = 4 * math.pi ** 2 * (k1 ** 2 + k2 ** 2)
        ksq[0, 0] = 1.0
        phi = torch.fft.fft2(rho - rho.mean()) / ksq
        phi[0, 0] = 0.0
        return [torch.fft.ifft2(-2j * math.pi * k * phi).real for k in (k1, k2)]

    def _evolve(self, J, dt):
        """One Yee step; E at the cell centres is the mean of before and after."""
        d1, d2 = self.pr.dq
        up1, up2 = (lambda a: a.roll(-1, 1)), (lambda a: a.roll(-1, 0))
        dn1, dn2 = (lambda a: a.roll(1, 1)), (lambda a: a.roll(1, 0))
        E1, E2, E3, B1, B2, B3 = self.yee
        E1 = E1 + dt * ((up2(B3) - B3) / d2 - J[0])
        E2 = E2 + dt * (-(up1(B3) - B3) / d1 - J[1])
        E3 = E3 + dt * ((up1(B2) - B2) / d1 - (up2(B1) - B1) / d2 - J[2])
        B1 = B1 - dt * (E3 - dn2(E3)) / d2
        B2 = B2 + dt * (E3 - dn1(E3)) / d1
        B3 = B3 - dt * ((E2 - dn1(E2)) / d1 - (E1 - dn2(E1)) / d2)
        self.yee = [E1, E2, E3, B1, B2, B3]
        now = [0.5 * (E1 + up1(E1)), 0.5 * (E2 + up2(E2)), E3, 0.5 * (B1 + up2(B1)),
               0.5 * (B2 + up1(B2)), 0.25 * (B3 + up2(B3) + up1(B3) + up1(up2(B3)))]
        self.cell = [0.5 * (a + b) for a, b in zip(self.cell[:3], now[:3])] + now[3:]

    def _bgk(self, f):
        p_dim, m = self.pr.p_dim, self.mass
        n = self._moment(f)
        u = [self._moment(f * v) / (n + 1e-30) for v in self.v]
        E = sum(self._moment(0.5 * f * v ** 2) for v in self.v)
        T = (2 * E * m - n * m * sum(x ** 2 for x in u)) / (n + 1e-30) / p_dim + 1e-30
        fm = n * (m / (2 * math.pi * T)) ** (p_dim / 2)
        for d in range(p_dim):
            fm = fm * torch.exp(-m * (self.v[d] - u[d]) ** 2 / (2 * T))
        return (fm - f) / TAU

    def _dfdt(self, f, evolve):
        c, pr = self.c, self.pr
        k, J = torch.zeros_like(f), []
        for axis, d in ((Q1, 0), (Q2, 1)):
            faces = f
            if pr.N[d] > 1:
                faces = _left_faces(f, axis, self.v[d], c['recon'], self.mirror)
                k -= _difference(self.v[d] * faces, axis) / pr.dq[d]
                faces = faces.narrow(axis, 0, pr.N[d])
            if evolve:
                J.append(self._charge_sum(self.v[d] * faces))
            del faces
        if c['source']:
            k += self._bgk(f)
        if c['fields'] == 'none':
            return k
        if c['fields'] == 'electrostatic':
            self.cell[:2] = self._poisson(f)
        elif evolve:
            self._evolve(J + [self._charge_sum(self.v[2] * f)], pr.dt)
        E1, E2, E3, B1, B2, B3 = [a[:, :, None, None, None, None] for a in self.cell]
        v1, v2, v3 = self.v
        em = self.charge / self.mass
        for d, (axis, a) in enumerate(((P1, em * (E1 + v2 * B3 - v3 * B2)),
                                       (P2, em * (E2 + v3 * B1 - v1 * B3)),
                                       (P3, em * (E3 + v1 * B2 - v2 * B1)))):
            if pr.P[d] > 1:
                k -= _difference(a * _left_faces(f, axis, a, c['recon']), axis) / pr.dp[d]
        return k

    def _advect(self, dt):
        """Every cell at the foot of its characteristic, Catmull-Rom in q1 and q2."""
        for axis, d in ((Q1, 0), (Q2, 1)):
            v, n = self.v[d].reshape(-1), self.pr.N[d]
            along = P1 if d == 0 else P2
            out = torch.empty_like(self.f)
            for i in range(v.numel()):
                shift = -float(v[i]) * dt / self.pr.dq[d]
                j = math.floor(shift)
                t = shift - j
                w = (-0.5 * t + t * t - 0.5 * t ** 3, 1 - 2.5 * t * t + 1.5 * t ** 3,
                     0.5 * t + 2 * t * t - 1.5 * t ** 3, -0.5 * t * t + 0.5 * t ** 3)
                f = self.f.select(along, i)
                out.select(along, i).copy_(sum(w[m] * f.roll(-(j - 1 + m), axis)
                                               for m in range(4)))
            self.f = out

    def step(self):
        f, dt = self.f, self.pr.dt
        if self.c['method'] == 'ASL':
            self._advect(0.5 * dt)
            f = self.f
            self.f = f + dt * self._bgk(f + 0.5 * dt * self._bgk(f))
            self._advect(0.5 * dt)
        elif self.c['integrator'] == 'RK2':
            x = f + 0.5 * dt * self._dfdt(f, False)
            self.f = f + dt * self._dfdt(x, True)
        else:
            k = self._dfdt(f, False)
            total = k.clone()
            for h, weight, evolve in ((0.5, 2, True), (0.5, 2, False), (1.0, 1, False)):
                k = self._dfdt(f + h * dt * k, evolve)
                total += weight * k
            self.f = f + dt / 6 * total

    def outputs(self):
        # (p, species, q1, q2), p1 fastest
        c = self.c
        out = dict(f=self.f.flatten(3).permute(3, 2, 1, 0))
        if c['N_q2'] == 1:
            out['density'] = self._moment(self.f)[..., 0, 0, 0].permute(2, 1, 0)[None]
        if c['fields'] == 'electrodynamic':
            out['fields'] = torch.stack(self.yee).permute(0, 2, 1)[:, None]
        return out


def _line_step(f, v, dp, dq, tau, dt):
    """One RK4 step of a 1D1V periodic run f (N_q1, N_p1) with BGK collisions."""
    def dfdt(f):
        g = f[torch.arange(-NG, f.shape[0] + NG, device=f.device) % f.shape[0]]
        n = f.shape[0] + 1
        win = lambda first: [g[first + t:first + t + n] for t in range(5)]
        F = v * torch.where(v > 0, _weno5(win(0), True), _weno5(win(1), False))
        rho = f.sum(1, keepdim=True) * dp
        u = (f * v).sum(1, keepdim=True) * dp / (rho + 1e-30)
        T = ((f * v * v).sum(1, keepdim=True) * dp - rho * u * u) / (rho + 1e-30) + 1e-30
        fm = rho * torch.sqrt(1 / (2 * math.pi * T)) * torch.exp(-(v - u) ** 2 / (2 * T))
        return -(F[1:] - F[:-1]) / dq - (f - fm) / tau
    k1 = dfdt(f)
    k2 = dfdt(f + 0.5 * dt * k1)
    k3 = dfdt(f + 0.5 * dt * k2)
    k4 = dfdt(f + dt * k3)
    return f + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def exact(case, seed):
    c = case
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    if c['path'] == 'solver':
        e = _Exact(c, seed)
        e.step()
        return e.outputs()
    if c['path'] == 'adjoint':
        f0, tau, dt = _rollout_inputs(c, seed)
        f0 = f0.to(dev).requires_grad_()
        tau = torch.tensor(tau, dtype=torch.float64, device=dev, requires_grad=True)
        n, dp = c['N_q1'], 12.0 / c['N_p1']
        v = -6.0 + (torch.arange(c['N_p1'], dtype=torch.float64, device=dev) + 0.5) * dp
        x = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n
        cos, sin = torch.cos(2 * math.pi * x), torch.sin(2 * math.pi * x)
        f, J = f0, 0.0
        for _ in range(c['steps']):
            f = _line_step(f, v, dp, 1.0 / n, tau, dt)
            rho = f.sum(1) * dp
            J = J + dt * (((rho * cos).mean()) ** 2 + ((rho * sin).mean()) ** 2)
        J.backward()
        return dict(J=J.detach(), f0=f0.grad, tau=tau.grad)
    done = []
    for r in _Sweep(c, seed).runs:
        n, dp = r['N_q1'], 20.0 / r['N_p1']
        v = -10.0 + (torch.arange(r['N_p1'], dtype=torch.float64, device=dev) + 0.5) * dp
        x = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n
        f = _Sweep.f0(r, x[:, None], v)
        for _ in range(c['steps']):
            f = _line_step(f, v, dp, 1.0 / n, r['tau'], r['dt'])
        done.append(f[torch.arange(-NG, n + NG, device=dev) % n].reshape(-1))
    return torch.cat(done)
