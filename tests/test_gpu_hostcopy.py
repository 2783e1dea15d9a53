"""GPU check of the copies between pageable host arrays and the device: arrays
below and above the size from which several threads copy, of one, two and
many buffer lengths with a remainder, and page-locked arrays, all move every
byte both ways; transfers from two host threads at once (one takes the
threads, the other the driver's copy) do too; and a state whose upload is
repeated gives the same steps, alone and in an ensemble."""
import threading

import numpy as np
import pytest

from helpers import cases, small_bubble

pytestmark = pytest.mark.gpu


def _round_trip(dcm, shape, seed, pinned=False):
    import torch

    kp, jp, ip = shape
    g = cases.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    core = dcm.DynamicalCore(g)
    rng = np.random.default_rng(seed)
    if pinned:
        t = torch.empty((ip + 2, jp + 2, kp + 2), dtype=torch.float64, pin_memory=True)
        a = t.numpy().transpose(2, 1, 0)
    else:
        a = np.empty((kp + 2, jp + 2, ip + 2), order="F")
    for _ in range(2):
        a[...] = rng.normal(size=a.shape)
        want = a.copy(order="F")
        # faces of k = 1..kp take their periodic images, the rest stays
        want[1:-1, 1:-1, 0], want[1:-1, 1:-1, -1] = want[1:-1, 1:-1, -2], want[1:-1, 1:-1, 1]
        want[1:-1, 0, 1:-1], want[1:-1, -1, 1:-1] = want[1:-1, -2, 1:-1], want[1:-1, 1, 1:-1]
        core.exchange_along_dim_wo(a)
        assert np.array_equal(a, want)
    core.close()


# 0.2, 2.1, 9, 17, 70 MB
SHAPES = [(30, 28, 26), (64, 62, 63), (104, 100, 103), (128, 126, 128), (128, 256, 256)]


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_whole_fields_both_ways(dcm, shape, pinned):
    _round_trip(dcm, shape, 81, pinned)


def test_two_threads(dcm):
    errors = []

    def go(seed):
        try:
            for n in range(3):
                _round_trip(dcm, SHAPES[2 + n % 2], seed + n)
        except BaseException as e:  # reported by the main thread
            errors.append(e)
    ts = [threading.Thread(target=go, args=(s,)) for s in (91, 92)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_repeated_upload_in_an_ensemble(dcm):
    """The captured steps are kept over an upload that changes no pointer and
    no configuration value, and made again when one changes."""
    cs = [small_bubble(), small_bubble(ip=20, jp=16, kp=12, seed=8)]
    ens = dcm.Ensemble([c.grid for c in cs])

    def leg(dt):
        for core, c in zip(ens.members, cs):
            core.upload_state(c.state, dt, ptol=c.ptol, kord=c.kord, precision=1)
            core.driver_start()
        ens.step(2)
        return [m.download_state() for m in ens.members]

    def alone(dt):
        out = []
        for c in cs:
            core = dcm.DynamicalCore(c.grid)
            core.upload_state(c.state, dt, ptol=c.ptol, kord=c.kord, precision=1)
            core.driver_start()
            core.step(2)
            out.append(core.download_state())
            core.close()
        return out
    for dt in (1.0, 1.0, 0.5, 1.0):
        for a, b in zip(leg(dt), alone(dt)):
            for n in ("u", "v", "w", "th", "p"):
                assert np.array_equal(a[n], b[n]), (dt, n)
    ens.close()
