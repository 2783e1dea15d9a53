"""GPU parity of the sedimentation calls' register form (kord 1, one halo level
in psi) against the oracle, at its dispatch's edges: levels that fill a lane's
registers and one more or less, the tallest column it takes and the next one
(which the general kernel takes), one to four fields, wider velocity halos,
per-column metrics and pass counts, the three Neumann options and an all-zero
column.  1e-12 relative max-norm per column and field, as the other drop-ins."""
import numpy as np
import pytest

from helpers import relerr
from test_oracle_column import _columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kp,nq,l_h,neumann", [
    (1, 1, 1, 0), (2, 2, 1, 1), (31, 3, 2, 2), (32, 2, 1, 0), (33, 1, 1, 1), (64, 3, 1, 0),
    (65, 2, 3, 2), (96, 1, 1, 0), (128, 2, 1, 0), (129, 3, 1, 1), (160, 2, 1, 0), (192, 1, 1, 2),
    (193, 3, 2, 0), (256, 2, 1, 0), (257, 2, 1, 0), (100, 4, 1, 0)])
def test_donor_cell_in_registers(dcm, orc, kp, nq, l_h, neumann):
    ncol = 11
    met, w, psi = _columns(700 + kp + nq, ncol, nq, kp, l_h, 1, kp % 2 == 1, zero_col=True)
    dt = np.linspace(0.5, 2.0, ncol)
    nsub = (1 + np.arange(ncol) % 4).astype(np.int32)
    a, b = psi.copy(), psi.copy()
    kw = dict(kord=1, monotone=False, neumann=neumann, l_h=l_h, r_h=1)
    dcm.mpdata_vec_1d_columns(dt, nsub, *met, w, a, **kw)
    orc.mpdata_vec_1d_columns(dt, nsub, *met, w, b, **kw)
    assert np.all(np.isfinite(a))
    for c in range(ncol):
        for n in range(nq):
            assert relerr(a[c, n], b[c, n]) <= 1e-12, (c, n)
