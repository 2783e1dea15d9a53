"""GPU check of the persistent FP64 preconditioner sweeps, taken once every
resident warp has eight warp tasks (64 k-levels of a row) or more: ragged rows and
levels, one to three k-chunks, a last pass over the tasks that only
some warps have.  The solve stops at ||r|| < tol max(||b||, 0.01)
(dynamics.f90:370-428); its solution's residual under the numpy operator is that
and the recursion's drift by round-off, far below tol = 1e-8."""
import numpy as np
import pytest

from helpers import cases, fz

pytestmark = pytest.mark.gpu


def _apply(g, x):
    c = x[1:-1, 1:-1, 1:-1]
    up = np.concatenate([c[1:], c[-1:]]) - c
    dn = np.concatenate([c[:1], c[:-1]]) - c
    d = float(g.dx[1]) ** 2
    return (up + dn + sum(np.roll(c, s, a) - c for a in (1, 2) for s in (-1, 1))) / d


@pytest.mark.parametrize("shape", [(201, 199, 6), (151, 131, 130), (257, 148, 66)])
def test_persistent_sweeps_solve(dcm, shape):
    ip, jp, kp = shape
    assert (kp + 63) // 64 * ip * jp >= 8 * 8 * 4 * 148  # tasks: the persistent form
    g = cases.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    rng = np.random.default_rng(72)
    b = fz(g)
    b[1:-1, 1:-1, 1:-1] = rng.normal(size=(kp, jp, ip))
    b[1:-1, 1:-1, 1:-1] -= b[1:-1, 1:-1, 1:-1].mean()
    x = fz(g)
    core = dcm.DynamicalCore(g)
    core.set_small_solver(0)
    it, err = core.bicgstab(x, b.copy(order="F"), fz(g), 1e-8)
    core.close()
    assert 0 < it and err < 1e-8
    res = b[1:-1, 1:-1, 1:-1] - _apply(g, x)
    assert np.sqrt(np.sum(res ** 2)) <= 2e-8 * max(np.sqrt(np.sum(b ** 2)), 0.01)
