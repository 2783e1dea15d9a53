"""GPU check of the quotients formed from tabled reciprocals (divergence_calc,
diagnostics.f90:120-153) where an infinity or a NaN enters: the same cells are
infinite, with the same sign, and the same are NaN as in the oracle's divisions;
the others agree to the tolerance of the other drop-in tests.  Zeros keep
their signs, and an infinite spacing gives a zero quotient."""
import numpy as np
import pytest

from helpers import cases, fz, rand_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("comp", [0, 1, 2])
def test_divergence_of_non_finite_velocities(dcm, orc, comp, value):
    g = cases.make_grid(9, 7, 35, 50.0, 60.0, 70.0, [-1.0e4, 1.0e5], [300.0, 310.0])
    rng = np.random.default_rng(26)
    f = [rand_field(g, rng) for _ in range(3)]
    f[comp][3, 4, 5] = value
    d1 = rand_field(g, rng)
    d2 = d1.copy(order="F")
    core, ocore = dcm.DynamicalCore(g), orc.OracleCore(g)
    core.divergence_calc(*f, d1)
    ocore.divergence_calc(*f, d2)
    core.close()
    assert np.count_nonzero(~np.isfinite(d2)) == 2
    assert np.array_equal(np.isnan(d1), np.isnan(d2))
    inf = np.isinf(d2)
    assert np.array_equal(np.isinf(d1), inf) and np.array_equal(d1[inf], d2[inf])
    ok = np.isfinite(d2)
    assert np.max(np.abs(d1[ok] - d2[ok])) <= 1e-12 * np.max(np.abs(d2[ok]))


def _divergence(dcm, g, u, v, w):
    d = fz(g)
    core = dcm.DynamicalCore(g)
    core.divergence_calc(u, v, w, d)
    core.close()
    return d[1:-1, 1:-1, 1:-1]


def test_quotients_keep_the_sign_of_zero(dcm, orc):
    g = cases.make_grid(9, 7, 35, 50.0, 60.0, 70.0, [-1.0e4, 1.0e5], [300.0, 310.0])
    f = [fz(g) for _ in range(3)]
    for a in f:
        a[3, 4, 5] = -0.0
    d = _divergence(dcm, g, *f)
    ref = fz(g)
    orc.OracleCore(g).divergence_calc(*f, ref)
    ref = ref[1:-1, 1:-1, 1:-1]
    assert np.count_nonzero(np.signbit(ref)) == 1
    assert np.array_equal(np.signbit(d), np.signbit(ref))


def test_quotients_by_an_infinite_spacing(dcm):
    g = cases.make_grid(9, 7, 35, 50.0, 60.0, 70.0, [-1.0e4, 1.0e5], [300.0, 310.0])
    g.dy[:] = g.dyn[:] = np.inf
    rng = np.random.default_rng(28)
    u, v, w = (rand_field(g, rng) for _ in range(3))
    assert np.array_equal(_divergence(dcm, g, u, v, w), _divergence(dcm, g, u, fz(g), w))
