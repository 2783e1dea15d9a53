"""GPU checks of the mixed form's direct corrections (transforms along x and y,
tridiagonal systems along z, in FP32, on the FP64 residual).

A step of domains above the size where they start, at transform lengths of
every kind (powers of two, products of the other small radices, primes alone
and with other radices, a length whose tiles are narrower, 1), columns of one to sixteen levels per
lane, odd level counts and stretched levels: the solve converges to ptol in a
handful of corrections, and the fields agree with the FP64 path's within the
mixed form's bars (1e-6 for p, whose right-hand side FP32 sources perturb;
1e-5 for the others).
"""
import ctypes

import numpy as np
import pytest

from helpers import cases, live_mask_p, relerr

pytestmark = pytest.mark.gpu


def _steps(dcm, c, precision, nsteps=2, graphs=1):
    core = dcm.DynamicalCore(c.grid)
    core.solver_graphs(graphs)
    core.upload_state(c.state, c.dt, ptol=c.ptol, kord=c.kord, precision=precision)
    core.driver_start()
    st = [core.step(1) for _ in range(nsteps)]
    f = core.download_state()
    core.close()
    return st, f


def _agree(c, f32, f64):
    m = live_mask_p(c.grid)
    p32, p64 = f32["p"][m], f64["p"][m]
    assert relerr(p32 - p32.mean(), p64 - p64.mean()) <= 1e-6
    for n in ("u", "v", "w", "th"):
        assert relerr(f32[n], f64[n]) <= 1e-5, n


SHAPES = [(64, 64, 48), (96, 60, 33), (97, 37, 61), (22, 91, 70), (26, 45, 128), (34, 127, 129),
          (320, 14, 40), (1, 640, 210), (800, 1, 257), (128, 9, 300)]


@pytest.mark.parametrize("shape", SHAPES)
def test_direct_corrections_match_the_fp64_path(dcm, shape):
    ip, jp, kp = shape
    c = cases.warm_bubble(ip=ip, jp=jp, kp=kp, dxyz=50.0, radius=400.0, zc=500.0, seed=61)
    st, f32 = _steps(dcm, c, 1)
    for s in st:
        assert s.err_last < c.ptol and 1 <= s.iters_last <= 5 and s.updates_last == s.iters_last
    _agree(c, f32, _steps(dcm, c, 0)[1])


def test_graph_and_host_driven_corrections_agree(dcm):
    c = cases.warm_bubble(ip=90, jp=50, kp=41, dxyz=50.0, radius=400.0, zc=500.0, seed=62)
    (sa, a), (sb, b) = (_steps(dcm, c, 1, graphs=g) for g in (1, 0))
    assert [s.iters_last for s in sa] == [s.iters_last for s in sb]
    for n in ("u", "v", "w", "th", "p"):
        assert np.array_equal(a[n], b[n]), n


def _with_spacing(g, axis, f):
    """The grid with its spacings along one axis (name "x" or "z") scaled by f."""
    for n in ("d" + axis, "d" + axis + "n"):
        setattr(g, n, getattr(g, n) * f)
    return g


@pytest.mark.parametrize("axis", ["z", "x"])
def test_stretched_spacings(dcm, axis):
    """Stretched levels keep the direct corrections (the tridiagonal systems
    take any spacing); uneven horizontal spacings take the FP32 iterations."""
    c = cases.warm_bubble(ip=72, jp=64, kp=40, dxyz=50.0, radius=400.0, zc=500.0, seed=63)
    n = len(getattr(c.grid, "d" + axis))
    q = np.arange(n) / (n - 1.0)
    _with_spacing(c.grid, axis,
                  1.0 + 0.5 * q if axis == "z" else 1.0 + 0.1 * np.sin(2 * np.pi * q))
    st, f32 = _steps(dcm, c, 1)
    assert all(s.err_last < c.ptol for s in st)
    assert all(s.iters_last <= 5 for s in st) if axis == "z" else \
        all(s.iters_last > 5 for s in st)
    _agree(c, f32, _steps(dcm, c, 0)[1])


def test_limits_of_the_direct_corrections(dcm):
    """itmax and the round budget bound the corrections as they bound the
    iterations, with the same statuses."""
    c = cases.warm_bubble(ip=64, jp=64, kp=48, dxyz=50.0, radius=400.0, zc=500.0, seed=64)
    core = dcm.DynamicalCore(c.grid)
    try:
        def fresh(itmax=9999):
            core.upload_state(c.state, c.dt, ptol=c.ptol, kord=c.kord, precision=1, itmax=itmax)
            core.driver_start()
        for itmax, rounds, status in ((1, 0, dcm.DCM_E_NOCONV), (9999, 1, dcm.DCM_E_TIMEOUT)):
            fresh(itmax)
            core.solver_limits(max_rounds=rounds)
            with pytest.raises(dcm.DCMError) as e:
                core.step(1)
            assert e.value.status == status
        core.solver_limits()
        fresh()
        assert core.step(1).err_last < c.ptol
    finally:
        core.close()


def _flat(shape, dx, dy, dz, mode=None, amp=0.0):
    """A bubble and noise on cells of dx, dy, dz, at rest; with mode, the
    starting pressure holds amp times that axis' longest wave."""
    ip, jp, kp = shape
    g = cases.make_grid(ip, jp, kp, dx, dy, dz, [-1.0e4, 1.0e5], [300.0, 300.0])
    rng = np.random.default_rng(65)
    r = np.sqrt((g.xn[None, None, 1:-1] / (0.2 * ip * dx)) ** 2 +
                (g.yn[None, 1:-1, None] / (0.2 * jp * dy)) ** 2 +
                ((g.zn[1:-1, None, None] - 0.5 * kp * dz) / (0.25 * kp * dz)) ** 2)
    th, p = cases.fzeros(kp, jp, ip), cases.fzeros(kp, jp, ip)
    th[1:-1, 1:-1, 1:-1] = 2.0 * np.cos(0.5 * np.pi * np.minimum(r, 1.0)) ** 2 + \
        rng.normal(0.0, 0.01, size=(kp, jp, ip))
    cases.exchange_full(th)
    if mode == "x":
        p[1:-1, 1:-1, 1:-1] = amp * np.cos(2 * np.pi * np.arange(ip) / ip)[None, None, :]
    st = cases.State(*(cases.fzeros(kp, jp, ip) for _ in range(9)), th, p)
    return g, st


# flat and oblong cells: 2^-24 times the operator's condition from 0.01 to 400
@pytest.mark.parametrize("shape,d", [
    ((256, 64, 40), (200.0, 200.0, 20.0)), ((256, 64, 40), (1000.0, 1000.0, 20.0)),
    ((256, 64, 40), (2000.0, 2000.0, 20.0)), ((256, 64, 40), (3000.0, 3000.0, 20.0)),
    ((256, 64, 40), (20000.0, 20000.0, 20.0)), ((97, 40, 70), (1000.0, 1000.0, 20.0)),
    ((64, 64, 130), (900.0, 900.0, 20.0)), ((64, 64, 300), (1500.0, 1500.0, 20.0)),
    ((256, 64, 40), (6000.0, 20.0, 20.0)), ((64, 256, 40), (20.0, 2000.0, 20.0)),
    ((3, 1500, 40), (20.0, 1000.0, 20.0))])
def test_flat_cells(dcm, shape, d):
    """Every solve converges, to the FP64 path's pressure within the mixed
    form's bar."""
    g, state = _flat(shape, *d)
    out = []
    for precision in (1, 0):
        core = dcm.DynamicalCore(g)
        core.upload_state(state, 1.0, ptol=1e-10, kord=3, precision=precision)
        core.driver_start()
        for _ in range(2):
            assert core.step(1).err_last < 1e-10
        out.append(core.download_state())
        core.close()
    p32, p64 = (f["p"][1:-1, 1:-1, 1:-1] for f in out)
    assert relerr(p32 - p32.mean(), p64 - p64.mean()) <= 1e-6


def test_pressure_is_put_back_for_the_iterations(dcm):
    """A correction that does not contract (flat cells, a starting pressure
    whose residual is the longest wave's) is undone: a round budget of that one
    correction ends the solve with the pressure it started with, and the
    iterations that follow are the same from a graph and from the host."""
    g, state = _flat((256, 64, 40), 1400.0, 1400.0, 20.0, "x", 1e5)
    out = []
    for graphs, itmax, rounds, status in ((1, 9999, 1, dcm.DCM_E_TIMEOUT),
                                          (1, 10, 0, dcm.DCM_E_NOCONV),
                                          (0, 10, 0, dcm.DCM_E_NOCONV)):
        core = dcm.DynamicalCore(g)
        core.solver_graphs(graphs)
        core.upload_state(state, 1.0, ptol=1e-10, kord=3, precision=1, itmax=itmax)
        core.driver_start()
        core.solver_limits(max_rounds=rounds)
        with pytest.raises(dcm.DCMError) as e:
            core.step(1)
        assert e.value.status == status
        out.append(core.download_state()["p"][1:-1, 1:-1, 1:-1])
        core.close()
    start = state.p[1:-1, 1:-1, 1:-1]
    assert np.array_equal(out[0], start)
    assert np.array_equal(out[1], out[2]) and not np.array_equal(out[1], start)


def _one_step(dcm, g, state, ptol, graphs=1, max_rounds=0):
    """(status, statistics, fields) of one mixed step, failed ones too."""
    core = dcm.DynamicalCore(g)
    core.solver_graphs(graphs)
    core.upload_state(state, 1.0, ptol=ptol, kord=3, precision=1)
    core.driver_start()
    core.solver_limits(max_rounds=max_rounds)
    s = dcm.StepStats()
    status = core.lib.dcm_step(core.h, 1, ctypes.byref(s))
    f = core.download_state()
    core.close()
    return status, s, f


def test_iterations_that_follow_a_correction_converge(dcm):
    """A starting pressure that is the longest wave alone, at rest: the first
    correction lowers its residual by less than a factor of 4, and the
    iterations take it below the tolerance (1e-3 of it), from a graph and from
    the host alike; the residual of the result is the one reported."""
    ip, jp, kp = 256, 64, 40
    g = cases.make_grid(ip, jp, kp, 600.0, 600.0, 20.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    p = cases.fzeros(kp, jp, ip)
    lam = (2.0 * np.sin(np.pi / ip) / 600.0) ** 2
    p[1:-1, 1:-1, 1:-1] = np.cos(2 * np.pi * np.arange(ip) / ip + 0.3)[None, None, :] / lam
    state = cases.State(*(cases.fzeros(kp, jp, ip) for _ in range(10)), p)
    start = np.sqrt(0.5 * ip * jp * kp) / 0.01  # ||A p|| / 0.01
    out = []
    for graphs in (1, 0):
        status, s, f = _one_step(dcm, g, state, 1e-3 * start, graphs)
        assert status == 0 and s.err_last < 1e-3 * start
        assert s.iters_last > 1 and s.iters_last != s.updates_last
        c = f["p"][1:-1, 1:-1, 1:-1]
        ax = (np.concatenate([c[1:], c[-1:]]) + np.concatenate([c[:1], c[:-1]]) - 2 * c) / 400.0
        ax += sum(np.roll(c, q, a) - c for a in (1, 2) for q in (-1, 1)) / 360000.0
        assert abs(np.sqrt(np.sum(ax ** 2)) / 0.01 - s.err_last) <= 1e-6 * s.err_last
        out.append((s.iters_last, s.updates_last, f))
    assert out[0][:2] == out[1][:2]
    for n in ("u", "v", "w", "p"):
        assert np.array_equal(out[0][2][n], out[1][2][n]), n


def test_iterations_that_follow_corrections_at_round_off(dcm):
    """A tolerance below what FP64 resolves: corrections until round-off, then
    the iterations up to itmax; the pressure stays what the corrections reached
    (the mixed form's bar against the FP64 path's)."""
    c = cases.warm_bubble(ip=64, jp=64, kp=33, dxyz=50.0, radius=400.0, zc=500.0, seed=66)
    core = dcm.DynamicalCore(c.grid)
    core.upload_state(c.state, c.dt, ptol=1e-20, kord=c.kord, precision=1, itmax=9)
    core.driver_start()
    s = dcm.StepStats()
    assert core.lib.dcm_step(core.h, 1, ctypes.byref(s)) == dcm.DCM_E_NOCONV
    assert s.iters_last >= 9 and 3 <= s.updates_last < s.iters_last
    m = (slice(1, -1),) * 3
    p = core.download_state()["p"][m]
    core.close()
    q = _steps(dcm, c, 0, nsteps=1)[1]["p"][m]
    assert relerr(p - p.mean(), q - q.mean()) <= 1e-6


def test_corrections_in_an_ensemble(dcm):
    """Members whose solves take direct corrections (one on flat cells, whose
    pressure is kept) beside one that iterates: the captured steps give the
    members' own, also over an upload that keeps them."""
    cs = [(c.grid, c.state, c.kord) for c in (
        cases.warm_bubble(ip=64, jp=64, kp=33, dxyz=50.0, radius=400.0, zc=500.0, seed=66),
        cases.warm_bubble(ip=24, jp=20, kp=16, dxyz=100.0, radius=500.0, zc=800.0, seed=67),
        cases.warm_bubble(ip=72, jp=50, kp=41, dxyz=50.0, radius=400.0, zc=500.0, seed=68))]
    cs.append(_flat((64, 64, 40), 4000.0, 4000.0, 20.0) + (3,))
    ens = dcm.Ensemble([c[0] for c in cs])

    def start(core, c):
        core.upload_state(c[1], 1.0, ptol=1e-10, kord=c[2], precision=1)
        core.driver_start()
    alone = []
    for c in cs:
        core = dcm.DynamicalCore(c[0])
        start(core, c)
        for _ in range(4):
            s = core.step(1)
        alone.append((s.iters_last, core.download_state()))
        core.close()
    assert [a[0] > 5 for a in alone] == [False, True, False, False]
    for _ in range(2):
        for core, c in zip(ens.members, cs):
            start(core, c)
        ens.step(4)
        for core, (_, f) in zip(ens.members, alone):
            g = core.download_state()
            for n in ("u", "v", "w", "th", "p"):
                assert np.array_equal(g[n], f[n]), n
    ens.close()


@pytest.mark.parametrize("graphs", [1, 0])
@pytest.mark.parametrize("value,size", [(np.inf, None), (1e200, 1e200)])
def test_corrections_end_at_an_infinite_residual(dcm, value, size, graphs):
    """A residual whose norm overflows contracts under no correction: after one
    the iterations take over, which end the step as they do without it."""
    c = cases.warm_bubble(ip=64, jp=64, kp=33, dxyz=50.0, radius=400.0, zc=500.0, seed=66)
    if size:
        c.state.p[1:-1, 1:-1, 1:-1] = size * np.random.default_rng(69).normal(size=(33, 64, 64))
    c.state.p[5, 6, 7] = value
    status, s, _ = _one_step(dcm, c.grid, c.state, 1e-10, graphs)
    assert status == dcm.DCM_E_NOCONV and s.iters_last <= 1 and np.isinf(s.err_last)
