"""Every stage kernel at the sizes where its tiling can go wrong: partial tiles
and chunks, rows off the vector width, one-cell axes, the smallest grids, and
the sizes at which another kernel takes over.

FP64 is compared with the FP64 oracle (the reference's operation order) to
1e-12 normwise, the tolerance of the parity tests: sums over at most 4e3 p-cells
in another order move a moment by 1e-16 sqrt(4e3), and the Maxwellian with it.
FP32 to 2e-6: 30 FP32 roundings (6e-8) per stage value.
"""

import numpy as np
import pytest
import torch

import cases as C
from _modules import make_solver, to_layout, moments_layout
from _util import interior, rel
from oracle.bolt_oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = {'fp64': 1e-12, 'fp32': 2e-6, 'fp64-fast': 1e-10}


def _spec(q, p, **kw):
    p_dim = 1 if p[1] == 1 else (2 if p[2] == 1 else 3)
    lim = [6.0 if n > 1 else 0.5 for n in p]
    base = dict(N_q1=q[0], N_q2=q[1], N_p1=p[0], N_p2=p[1], N_p3=p[2], p_dim=p_dim,
                mass=[1.0], charge=[-1.0], tau=0.05, dt=5e-4, steps=2, integrator='RK2',
                init=dict(amp=0.1, k1=1, k2=1 if q[1] > 1 else 0, noise=1e-2, seed=5,
                          u=[0.2, -0.1, 0.1]))
    ns = len(kw.get('mass', base['mass']))
    for d in range(3):
        base['p%d_start' % (d + 1)] = [-lim[d]] * ns
        base['p%d_end' % (d + 1)] = [lim[d]] * ns
    base.update(kw)
    return C.make(**base)


def _steps(nls, spec):
    for _ in range(spec['steps']):
        nls.strang_timestep(spec['dt'])


def _against_oracle(spec, precision, fields=False):
    nls = make_solver(spec, precision)
    o = Oracle(spec, to_layout(nls.f, spec))
    if fields and spec['fields_type'] == 'electrodynamic':
        o.fields.cell = nls.fields_solver.cell_centered_EM_fields[:, 0].permute(0, 2, 1).cpu().numpy()
        o.fields.yee = nls.fields_solver.yee_grid_EM_fields[:, 0].permute(0, 2, 1).cpu().numpy()
    for _ in range(spec['steps']):
        nls.strang_timestep(spec['dt'])
        o.step(spec['dt'])
    g = spec['N_ghost']
    assert rel(interior(to_layout(nls.f, spec), g), interior(o.f, g)) < TOL[precision]
    for k in ('density', 'energy'):
        got = interior(moments_layout(nls.compute_moments(k)), g)
        assert rel(got, interior(o.moments(k), g)) < TOL[precision]
    return nls, o


# sizes around the 8x8 q-tile and the 32-wide p-chunk: below, at and above them
SIZES = [((6, 6), (5, 4, 3)), ((7, 9), (8, 4, 1)), ((8, 8), (16, 3, 2)), ((9, 16), (31, 1, 3)),
         ((17, 8), (33, 3, 1)), ((15, 15), (12, 11, 5))]


@pytest.mark.parametrize('precision', ['fp64', 'fp32', 'fp64-fast'])
@pytest.mark.parametrize('q,p', SIZES)
@pytest.mark.parametrize('integrator', ['RK2', 'RK4'])
def test_any_grid(q, p, precision, integrator):
    """Fused stages (with the source) on grids off the tiles."""
    _against_oracle(_spec(q, p, integrator=integrator), precision)


@pytest.mark.parametrize('recon', ['minmod', 'ppm', 'piecewise-constant'])
@pytest.mark.parametrize('bc', ['periodic', 'mirror'])
def test_any_grid_reconstructions_and_walls(recon, bc):
    _against_oracle(_spec((11, 10), (9, 6, 2), recon_q=recon, bc_q1=bc, bc_q2=bc), 'fp64')


@pytest.mark.parametrize('q,p', [((8, 16), (8, 4, 3)), ((16, 8), (16, 2, 1)), ((9, 7), (15, 5, 1))])
@pytest.mark.parametrize('source', [False, True])
def test_tile_kernels_write_the_scalar_kernels_bits(monkeypatch, q, p, source):
    """FP64 in the reference's operation order: the tile kernels and the scalar
    kernel (BOLT_NO_PAIR) do the same operations per value, so one step without
    the source agrees bit for bit, and with it up to the order of the moments'
    partial sums."""
    out = []
    for off in (False, True):
        if off:
            monkeypatch.setenv('BOLT_NO_PAIR', '1')
        nls = make_solver(_spec(q, p, source_enabled=source, integrator='RK4'), 'fp64')
        nls.strang_timestep(5e-4)
        out.append(nls.f.cpu().numpy())
    if source:
        assert rel(out[0], out[1]) < 1e-14
    else:
        assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize('q,p', [((9, 8), (33, 3, 1)), ((16, 16), (8, 4, 2))])
@pytest.mark.parametrize('chunks', [None, '1'])
def test_currents_write_the_scalar_kernels_bits(monkeypatch, q, p, chunks):
    """FP64 currents by the tile kernel and by the scalar kernel, split the same
    way: the fields they drive have the same bits, also where a CTA's first chunk
    of p is its only one, in every run."""
    if chunks:
        monkeypatch.setenv('BOLT_CHUNKS_PER_SPLIT', chunks)
    spec = _spec(q, p, fields_enabled=True, source_enabled=False, integrator='RK4')

    def fields():
        nls = make_solver(spec, 'fp64')
        nls.strang_timestep(5e-4)
        return nls.fields_solver.yee_grid_EM_fields.cpu().numpy()
    tiles = [fields() for _ in range(8)]
    monkeypatch.setenv('BOLT_NO_PAIR', '1')
    scalar = fields()
    assert np.abs(scalar).max() > 0
    for t in tiles:
        assert np.array_equal(t, scalar)


# p-blocks: one-cell axes, two cells (the window wraps onto itself), rows of one
# vector and off it, more lines than threads
PBLOCKS = [(8, 1, 1), (2, 3, 1), (1, 5, 4), (5, 2, 3), (4, 4, 4), (33, 7, 1), (12, 11, 10)]


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('p', PBLOCKS)
@pytest.mark.parametrize('recon', ['weno5', 'minmod'])
def test_p_stage_blocks(p, precision, recon):
    spec = _spec((8, 7), p, fields_enabled=True, recon_q=recon, recon_p=recon,
                 mass=[1.0, 2.0], charge=[-1.0, 1.5], p_dim=max(1, sum(n > 1 for n in p)))
    spec['p_dim'] = 3 if p[2] > 1 else (2 if p[1] > 1 else 1)
    nls, o = _against_oracle(spec, precision, fields=True)
    got = nls.fields_solver.yee_grid_EM_fields[:, 0].permute(0, 2, 1).cpu().numpy()
    assert rel(interior(got.transpose(1, 2, 0), 3), interior(o.fields.yee.transpose(1, 2, 0), 3)) \
        < (1e-10 if precision == 'fp64' else 1e-4)


@pytest.mark.parametrize('N,N_p1,cells', [(6, 24, 1), (7, 24, 1), (64, 24, 1), (129, 24, 1),
                                          (601, 130, 2), (1003, 201, 4), (2048, 24, 1),
                                          (2049, 24, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_electrostatic_line(N, N_p1, cells, precision):
    """N_q2 = 1: E1 from the Green's function of the periodic solve, even and odd
    lines (the Nyquist mode of an even one drops out), up to 2,048 cells and, past
    them, from the FFT; the q-part by the line kernel at each of its forms."""
    spec = _spec((N, 1), (N_p1, 1, 1), fields_enabled=True, fields_type='electrostatic',
                 fields_solver='fft', source_enabled=False, dt=5e-4 if N < 200 else 0.1 / N / 6)
    nls, o = _against_oracle(spec, precision, fields=True)
    _line_cells(nls, cells)
    got = nls.fields_solver.cell_centered_EM_fields[:2, 0].permute(0, 2, 1).cpu().numpy()
    assert rel(got, o.fields.cell[:2]) < (1e-11 if precision == 'fp64' else 1e-5)


# 1D1V: 1, 2 and 4 q-cells per thread of the line kernel (148 SMs), partial last
# groups, p below, at and above the CTA's threads, one and two species; 0: the sizes
# just past it and well past it, on the scalar kernel's tiles
LINES = [(6, 5, 1), (9, 32, 1), (64, 300, 1), (601, 130, 2), (1003, 201, 4), (1183, 256, 4),
         (1184, 256, 0), (1201, 512, 0)]


def _line_cells(nls, cells):
    assert nls._lib.bolt_line_cells(nls._ctx) == cells


@pytest.mark.parametrize('N_q1,N_p1,cells', LINES)
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('source', [False, True])
def test_line(N_q1, N_p1, cells, precision, source):
    ns = 2 if N_q1 < 100 else 1
    nls, _ = _against_oracle(_spec((N_q1, 1), (N_p1, 1, 1), source_enabled=source,
                                   mass=[1.0, 2.0][:ns], charge=[0.0] * ns,
                                   dt=0.1 / N_q1 / 6), precision)
    _line_cells(nls, cells)


@pytest.mark.parametrize('precision,cells', [('fp64', 4), ('fp32', 0)])
def test_line_waves(precision, cells):
    """Two waves of CTAs of the line kernel: taken in FP64, not in FP32."""
    nls, _ = _against_oracle(_spec((4062, 1), (64, 1, 1), dt=0.1 / 4062 / 6), precision)
    _line_cells(nls, cells)


@pytest.mark.parametrize('tau', [float('inf'), 1e-2])
@pytest.mark.parametrize('q,p', [((32, 1), (40, 1, 1)), ((8, 8), (8, 4, 1)), ((9, 8), (8, 3, 1))])
def test_infinite_collision_time(q, p, tau):
    """tau = inf divides the source to zero in every kernel."""
    spec = _spec(q, p, tau=tau)
    nls, o = _against_oracle(spec, 'fp64')
    if tau == float('inf'):
        assert bool(torch.isfinite(nls.f).all())


@pytest.mark.parametrize('q,p', [((64, 64), (16, 16, 1)), ((21, 21), (33, 8, 1)),
                                 ((1000, 1), (96, 1, 1))])
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('integrator', ['RK2', 'RK4'])
def test_kernels_take_turns(q, p, precision, integrator):
    """Steps by the grid's own kernel and, with a tau array, by the scalar one, a
    df/dt in between: each is cut for itself, so a stage may find another number of
    partial moment sums than it leaves."""
    spec = _spec(q, p, integrator=integrator, dt=1e-4)
    nls = make_solver(spec, precision)
    o = Oracle(spec, to_layout(nls.f, spec))
    lib, ctx = nls._lib, nls._ctx
    tau = torch.full_like(nls._fstore, spec['tau'])
    for array in (False, True, True, False):
        lib.bolt_set_tau_array(ctx, tau.data_ptr() if array else None)
        nls.strang_timestep(spec['dt'])
        o.step(spec['dt'])
        out = torch.empty_like(nls._fstore)
        assert lib.bolt_dfdt(ctx, nls._fstore.data_ptr(), out.data_ptr(), 0, 0.0, nls._stream()) == 0
    nls.synchronize()
    g = spec['N_ghost']
    assert rel(interior(to_layout(nls.f, spec), g), interior(o.f, g)) < TOL[precision]


@pytest.mark.parametrize('p', [(8, 6, 4), (7, 5, 3), (30, 1, 1)])
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_semi_lagrangian_source_blocks(p, precision):
    """The source's RK2 step with the p-block in shared memory, rows on and off
    the 16-byte vectors, against the oracle's."""
    spec = _spec((9, 8), p, solver_q='ASL', integrator='RK4')
    nls = make_solver(spec, precision)
    o = Oracle(spec, to_layout(nls.f, spec))
    for _ in range(2):
        nls.lie_timestep(spec['dt'])
        o.split_step(spec['dt'], 'lie')
    g = spec['N_ghost']
    assert rel(interior(to_layout(nls.f, spec), g), interior(o.f, g)) < TOL[precision]


@pytest.mark.parametrize('n', [(64, 64), (122, 122), (123, 122), (250, 251)])
def test_field_update_by_cluster_or_by_passes(n):
    """One update with given currents on grids below, at and above the size
    (2^14 cells with the ghosts) at which the passes become launches."""
    spec = _spec(n, (2, 2, 1), fields_enabled=True, source_enabled=False)
    nls = make_solver(spec, 'fp64')
    o = Oracle(spec, to_layout(nls.f, spec))
    rng = np.random.default_rng(2)
    y = rng.standard_normal(o.fields.yee.shape)
    af = lambda a: torch.from_numpy(a.copy()).permute(0, 2, 1).unsqueeze(1).cuda()
    nls.fields_solver.yee_grid_EM_fields = af(y)
    o.fields.yee = y.copy()
    o.fields.cell = nls.fields_solver.cell_centered_EM_fields[:, 0].permute(0, 2, 1).cpu().numpy()
    J = rng.standard_normal((3,) + y.shape[1:])
    nls.fields_solver.evolve_electrodynamic_fields(*[af(J[k:k + 1]) for k in range(3)], 1e-3)
    o.fields.evolve(J[0], J[1], J[2], 1e-3)
    for got, want in ((nls.fields_solver.yee_grid_EM_fields, o.fields.yee),
                      (nls.fields_solver.cell_centered_EM_fields, o.fields.cell)):
        got = got[:, 0].permute(0, 2, 1).cpu().numpy()
        assert rel(got, want) < 1e-14


@pytest.mark.parametrize('N_q1,N_p1', [(6, 33), (7, 257), (33, 600)])
@pytest.mark.parametrize('recon', ['weno5', 'minmod'])
def test_adjoint_rows(N_q1, N_p1, recon):
    """The smallest lines (a window wraps around them) and rows longer than the
    CTA: gradients against autograd of the transcription."""
    from bolt_b200.adjoint import Rollout1D1V
    from oracle.bolt_torch import Problem1D1V
    dt, tau, steps = 0.1 / N_q1 / 6, 0.03, 6
    q = (torch.arange(N_q1, dtype=torch.float64, device='cuda') + 0.5) / N_q1
    p = -6 + (torch.arange(N_p1, dtype=torch.float64, device='cuda') + 0.5) * 12 / N_p1
    f0 = (1 + 0.2 * torch.cos(2 * np.pi * q))[:, None] * torch.exp(-(p - 0.3) ** 2 / 2)[None]
    r = Rollout1D1V(N_q1, N_p1, -6.0, 6.0, dt, tau, steps, snapshots=2, reconstruction=recon)
    gf, gt = r.gradient(f0)
    pr = Problem1D1V(N_q1, N_p1, -6.0, 6.0, dt, tau, device='cuda', **(
        {} if recon == 'weno5' else {'reconstruction': recon}))
    x, t = f0.clone().requires_grad_(), torch.tensor(tau, dtype=torch.float64, device='cuda',
                                                      requires_grad=True)
    J, _ = pr.objective(x, t, steps)
    J.backward()
    # the derivatives of the WENO weights amplify rounding by up to 1/beta
    assert rel(gf.cpu(), x.grad.cpu()) < 1e-9
    assert abs(float(gt) - float(t.grad)) < 1e-8 * abs(float(t.grad)) + 1e-15
