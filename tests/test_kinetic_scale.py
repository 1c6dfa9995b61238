"""The kinetic step's change of psi in complex64 carries 1/N to more than one FP32 word.

On these grids that word alone is 5.2e-8 to 5.8e-8 above 1/N, one-sided on every increment.  The
increments are projected on FP64's: roundings of single points average out over 1e5 points and more,
those of the phase tables over dozens of entries an axis (a few 1e-9 to 1.4e-8).  Bound: half of the
smallest word error, 2.6e-8."""
import numpy as np
import pytest

import gpesolver_b200 as G
from oracle import oracle as O

from .helpers import gparams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(128, 126, 32), (126, 98, 42), (128, 81, 49)])
def test_increment_is_not_scaled_by_a_rounded_1_over_n(dims):
    n = dims[0] * dims[1] * dims[2]
    assert abs(float(np.float32(1 / n)) * n - 1) > 5.2e-8
    p = gparams(O.default_config(nx=dims[0], ny=dims[1], nz=dims[2]))
    rng = np.random.default_rng(1)
    psi = rng.normal(size=dims) + 1j * rng.normal(size=dims)
    psi /= np.sqrt((np.abs(psi) ** 2).sum() * p.dx * p.dy * p.dz)
    psi = psi.astype(np.complex64).astype(np.complex128)
    with G.B200GrossPitaevskiSolver(p, precision="c64", schedule="split") as s:
        s.import_data(psi)
        s.real_fft_kinetic_step()
        got = s.export_data() - psi
    q = [2 * np.pi * np.fft.fftfreq(m, d) for m, d in zip(dims, (p.dx, p.dy, p.dz))]
    q2 = q[0][:, None, None] ** 2 + q[1][None, :, None] ** 2 + q[2] ** 2
    want = np.fft.ifftn(np.fft.fftn(psi) * np.expm1(-1j * p.real_time_dt / (2 * p.m) * q2))
    assert abs((np.vdot(want, got) / np.vdot(want, want)).real - 1) < 2.6e-8
