"""States far from the smooth, order-one ones of the other tests: jumps of large
values beside exactly uniform data, values whose squares leave the range, and steps as
long as the collision time."""

import os
import sys

import numpy as np
import pytest
import torch

import cases as C
from _modules import make_solver, to_layout
from _util import interior, rel
from oracle.bolt_oracle import Oracle
from test_gpu_kernel_sizes import TOL, _spec
from test_gpu_parity import af_from_layout

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

pytestmark = pytest.mark.gpu


def _from(spec, precision, f0):
    """A solver and an oracle holding f0, given in the oracle's layout."""
    nls = make_solver(spec, precision)
    f0 = f0.astype(np.float32).astype(np.float64)
    nls.f = af_from_layout(f0).to('cuda')
    return nls, Oracle(spec, f0)


def _steps(nls, o, spec):
    for _ in range(spec['steps']):
        nls.strang_timestep(spec['dt'])
        o.step(spec['dt'])
    g = spec['N_ghost']
    return interior(to_layout(nls.f, spec), g), interior(o.f, g)


def _q_jump(spec, top):
    """Two uniform halves along q1, every cell a Maxwellian of the same width."""
    o = Oracle(spec, to_layout(make_solver(spec, 'fp64').f, spec))
    cell = o.f[spec['N_ghost'], spec['N_ghost']]
    i = np.arange(o.f.shape[1]) - spec['N_ghost']
    half = (i % spec['N_q1']) < spec['N_q1'] // 2
    return np.broadcast_to(np.where(half, top, 0.125 * top)[None, :, None, None, None, None]
                           * cell, o.f.shape).copy()


# With a smoothness indicator's floor of 1e-17 the weight of a uniform substencil
# is 1e34: times the third difference across a jump beyond 3e4 it leaves FP32, though
# the face value does not
@pytest.mark.parametrize('top', [1e2, 1e6, 1e9])
@pytest.mark.parametrize('integrator', ['RK2', 'RK4'])
def test_jump_in_q(top, integrator):
    spec = _spec((21, 10), (9, 6, 2), source_enabled=False, integrator=integrator)
    got, want = _steps(*_from(spec, 'fp32', _q_jump(spec, top)), spec)
    assert rel(got, want) < TOL['fp32']


@pytest.mark.parametrize('top', [1e2, 1e6, 1e9])
@pytest.mark.parametrize('p', [(20, 1, 1), (16, 12, 1), (9, 8, 10)])
def test_jump_in_p(top, p):
    """A block of a uniform value in velocity space, empty around it, in the
    field of its density wave."""
    spec = _spec((9, 10), p, source_enabled=False, fields_enabled=True,
                 fields_type='electrostatic', fields_solver='fft', charge=[-1.0 / top])
    o = Oracle(spec, to_layout(make_solver(spec, 'fp64').f, spec))
    f0 = np.zeros(o.f.shape)
    inner = tuple(slice(n // 4, n - n // 4) for n in reversed(p))
    wave = top * (1 + 0.1 * np.cos(2 * np.pi * (np.arange(f0.shape[1]) - 2.5) / 9))
    f0[(Ellipsis,) + inner] = wave[None, :, None, None, None, None]
    nls, o = _from(spec, 'fp32', f0)
    got, want = _steps(nls, o, spec)
    assert rel(got, want) < TOL['fp32']


@pytest.mark.parametrize('top', [1e2, 1e6, 1e9])
def test_jump_in_a_batch(top):
    from bolt_b200.batch import BatchSolver
    r = dict(N_q1=32, N_p1=64, tau=0.01, amp=0.0, k=1, dt=0.5 / 32 / 10.0)
    bs = BatchSolver([bench.ragged_system(r, source=False)], [r['dt']])
    f = bs.f(0)
    half = (torch.arange(f.shape[2], device=f.device) - 3) % 32 < 16
    f.mul_(torch.where(half, top, 0.125 * top)[None, None, :, None])
    spec = C.make(N_q1=32, N_q2=1, N_p1=64, N_p2=1, N_p3=1, p1_start=[-10.0], p1_end=[10.0],
                  p2_start=[-0.5], p2_end=[0.5], p3_start=[-0.5], p3_end=[0.5], mass=[1.0],
                  charge=[0.0], p_dim=1, dt=r['dt'], integrator='RK4', source_enabled=False,
                  init=dict(amp=0.0, k1=1, k2=0))
    q1p = f[:, 0, :, 0].double().T.cpu().numpy()
    o = Oracle(spec, np.ascontiguousarray(np.broadcast_to(
        q1p[None, :, None, None, None, :], (7,) + q1p.shape[:1] + (1, 1, 1) + q1p.shape[1:])))
    bs.run(3)
    bs.synchronize()
    for _ in range(3):
        o.step(r['dt'])
    got = bs.f(0)[:, 0, :, 0].double().T.cpu().numpy()[3:-3]
    assert rel(got, o.f[3, 3:-3, 0, 0, 0, :]) < TOL['fp32']


KERNELS = [dict(q=(32, 1), p=(40, 1, 1)),                          # line
           dict(q=(16, 16), p=(8, 4, 1)),                          # whole tiles
           dict(q=(9, 10), p=(9, 4, 1)),                           # any grid
           dict(q=(9, 10), p=(9, 4, 1), scalar=True),
           dict(q=(9, 10), p=(16, 6, 1), fields=True)]             # p-stage


def _large_state(kernel, monkeypatch, fn):
    if kernel.get('scalar'):
        monkeypatch.setenv('BOLT_NO_PAIR', '1')
    kw = dict(fields_enabled=True, fields_type='electrostatic', fields_solver='fft',
              charge=[-1e-170]) if kernel.get('fields') else {}
    spec = _spec(kernel['q'], kernel['p'], source_enabled=False, steps=1, **kw)
    nls = make_solver(spec, 'fp64')
    f0 = fn(to_layout(nls.f, spec))
    nls.f = af_from_layout(f0).to('cuda')
    return spec, nls, Oracle(spec, f0)


@pytest.mark.parametrize('kernel', KERNELS)
def test_reference_order_diverges_where_the_reference_does(monkeypatch, kernel):
    """The smoothness indicators' squares overflow for noise of 1e90: every weight of
    the reference is zero, its face 0/0, and the run stops."""
    rng = np.random.default_rng(3)
    spec, nls, o = _large_state(kernel, monkeypatch,
                                lambda f: 1e90 * (1 + rng.random(f.shape)))
    with np.errstate(all='ignore'), pytest.raises(SystemExit):
        o.step(spec['dt'])
    with pytest.raises(SystemExit):
        for _ in range(2):                # the flag of a step is read by the next one
            nls.strang_timestep(spec['dt'])
            torch.cuda.synchronize()


@pytest.mark.parametrize('kernel', KERNELS)
@pytest.mark.parametrize('top', [1e60, 1e90])
def test_reference_order_beside_a_huge_value(monkeypatch, kernel, top):
    """One value of `top`: at 1e90 the squares of its substencils overflow, faces
    with nothing else are NaN, and the ones with an ordinary substencil keep to it."""
    rng = np.random.default_rng(4)

    def state(f):
        f = f * (1 + 0.1 * rng.random(f.shape))
        f[:, 3 + 4, 0, 0, 1 if f.shape[4] > 1 else 0, 5] = top
        return f
    spec, nls, o = _large_state(kernel, monkeypatch, state)
    with np.errstate(all='ignore'):
        o.fvm_step(spec['dt'])
    nls.strang_timestep(spec['dt'])
    g = spec['N_ghost']
    got, want = interior(to_layout(nls.f, spec), g), interior(o.f, g)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.isfinite(want).all() == (top == 1e60)
    small = np.isfinite(want) & (np.abs(want) < 10)
    if kernel.get('fields') and top == 1e90:
        assert not small.any()                 # the Poisson solve spreads a NaN
        return
    assert small.sum() > 0.5 * want.size
    assert rel(got[small], want[small]) < TOL['fp64']


@pytest.mark.parametrize('q,p', [((11, 13), (15, 13, 14)), ((9, 10), (20, 18, 1)), ((20, 1), (60, 1, 1))])
@pytest.mark.parametrize('fields', [False, True])
def test_stiff_source(q, p, fields):
    """dt = tau in FP32, off the whole tiles: RK2 keeps half of f's error and adds the
    rounding of two stored stages (3.4e-8 rms each), 5.5e-8 in all at worst; a Maxwellian
    of rounded factors would double that after ten steps."""
    kw = dict(fields_enabled=True, fields_type='electrostatic', fields_solver='fft',
              charge=[-0.1]) if fields else {}
    spec = _spec(q, p, dt=1e-3, tau=1e-3, steps=30, **kw)
    nls = make_solver(spec, 'fp32')
    o = Oracle(spec, to_layout(nls.f, spec))
    got, want = _steps(nls, o, spec)
    assert rel(got, want) < 1e-7
