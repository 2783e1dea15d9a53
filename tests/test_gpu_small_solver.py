"""GPU check of the one-point-per-thread cluster solve of small FP64 domains
against the multi-kernel solve: domains that fill the cluster's threads
exactly, one point more than a block, ragged last blocks, single rows and
single planes, neighbours that wrap onto the point itself.  Both stop at
||r|| < tol max(||b||, 0.01) (dynamics.f90:370-428), so the residuals of the two
solutions under the numpy operator are below tol and the difference of the
solutions is at most the sum of two such errors."""
import numpy as np
import pytest

from helpers import cases, fz, rand_field

pytestmark = pytest.mark.gpu


def _residual(g, x, b):
    c = x[1:-1, 1:-1, 1:-1]
    up = np.concatenate([c[1:], c[-1:]]) - c
    dn = np.concatenate([c[:1], c[:-1]]) - c
    d = float(g.dx[1]) ** 2
    ax = up + dn + sum(np.roll(c, s, a) - c for a in (1, 2) for s in (-1, 1))
    return b[1:-1, 1:-1, 1:-1] - ax / d


@pytest.mark.parametrize("shape", [(128, 1, 64), (1, 128, 64), (27, 19, 8), (171, 1, 3),
                                   (19, 9, 3), (2, 2, 5), (16, 16, 31), (1, 1, 513)])
def test_point_solver_matches_the_multi_kernel_solve(dcm, shape):
    ip, jp, kp = shape
    assert ip * jp * kp <= 8192
    g = cases.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    rng = np.random.default_rng(71)
    b = fz(g)
    b[1:-1, 1:-1, 1:-1] = rng.normal(size=(kp, jp, ip))
    b[1:-1, 1:-1, 1:-1] -= b[1:-1, 1:-1, 1:-1].mean()
    x0 = rand_field(g, rng, -0.01, 0.01)
    core = dcm.DynamicalCore(g)
    out = []
    for small in (8192, 0):
        core.set_small_solver(small)
        x = x0.copy(order="F")
        it, err = core.bicgstab(x, b.copy(order="F"), fz(g), 1e-10)
        assert 0 < it and err < 1e-10
        out.append((it, x))
    core.close()
    sc = max(np.sqrt(np.sum(b[1:-1, 1:-1, 1:-1] ** 2)), 0.01)
    for _, x in out:
        # the recursion's residual drifts from the true one by round-off
        assert np.sqrt(np.sum(_residual(g, x, b) ** 2)) <= 2e-10 * sc
    # sums in another order: the recursions part by round-off
    assert abs(out[0][0] - out[1][0]) <= 3 + 0.05 * out[1][0]


def _system(shape):
    ip, jp, kp = shape
    g = cases.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    rng = np.random.default_rng(71)
    b = fz(g)
    b[1:-1, 1:-1, 1:-1] = rng.normal(size=(kp, jp, ip))
    b[1:-1, 1:-1, 1:-1] -= b[1:-1, 1:-1, 1:-1].mean()
    return g, b, rand_field(g, rng, -0.01, 0.01)


SHAPES = [(128, 1, 64), (1, 128, 64), (27, 19, 8), (171, 1, 3), (19, 9, 3), (2, 2, 5),
          (16, 16, 31), (1, 1, 513)]


@pytest.mark.parametrize("shape", SHAPES)
def test_clusters_of_8_and_16_blocks_give_the_same_bits(dcm, shape):
    g, b, x0 = _system(shape)
    core = dcm.DynamicalCore(g)
    out = []
    for blocks in (16, 8):
        core.set_small_cluster(blocks)
        x = x0.copy(order="F")
        out.append((core.bicgstab(x, b.copy(order="F"), fz(g), 1e-10), x))
    core.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("shape", [(129, 1, 64), (31, 29, 37), (64, 40, 9)])
def test_larger_domains_in_one_cluster(dcm, shape):
    """Above 8192 points, with the limit raised: more than one point a thread."""
    g, b, x0 = _system(shape)
    assert 8192 < np.prod(shape) < 65536
    core = dcm.DynamicalCore(g)
    sc = max(np.sqrt(np.sum(b[1:-1, 1:-1, 1:-1] ** 2)), 0.01)
    its = []
    for small in (65536, 0):
        core.set_small_solver(small)
        x = x0.copy(order="F")
        it, err = core.bicgstab(x, b.copy(order="F"), fz(g), 1e-10)
        assert 0 < it and err < 1e-10
        assert np.sqrt(np.sum(_residual(g, x, b) ** 2)) <= 2e-10 * sc
        its.append(it)
    core.close()
    assert abs(its[0] - its[1]) <= 3 + 0.05 * its[1]
