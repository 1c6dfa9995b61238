"""Every radix and stage count of the run-time line transforms (general.cuh): the
dipolar field and one kinetic step against numpy's FFTs, at sizes where a tile, a row
pair or a line is ragged, and with lines of one point.

Tolerances: complex128, 1e-13 (a few roundings of 1e-16 a stage); complex64, 1e-6 (a
stage's rounding is 6e-8, compensated twiddles add none of their own; about ten
stages there and back)."""
import numpy as np
import pytest

import gpesolver_b200 as G
from oracle import oracle as O

from .helpers import gparams, rel_l2

pytestmark = pytest.mark.gpu

DIMS = [(5, 7, 3), (1, 9, 12), (21, 1, 10), (14, 15, 1), (27, 6, 4), (49, 35, 9), (50, 45, 14), (125, 12, 5),
        (81, 10, 16), (24, 100, 30), (16, 96, 25), (3, 250, 7), (343, 4, 8), (10, 18, 100), (2, 2, 2), (144, 21, 20)]


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("dims", DIMS)
def test_lines_match_numpy(dims, prec):
    nx, ny, nz = dims
    p = gparams(O.default_config(nx=nx, ny=ny, nz=nz))
    rng = np.random.default_rng(nx * ny + nz)
    psi = rng.normal(size=dims) + 1j * rng.normal(size=dims)
    psi /= np.sqrt((np.abs(psi) ** 2).sum() * p.dx * p.dy * p.dz)
    with G.B200GrossPitaevskiSolver(p, precision=prec, schedule="split") as s:
        s.load_buffer(psi)
        s.calc_fi3d()
        phi = s.export_fi3d()
        s.real_fft_kinetic_step()
        out = s.export_data()
        n = s.calc_norm()
    k = [2 * np.pi * np.fft.fftfreq(2 * m, d) for m, d in zip(dims, (p.dx, p.dy, p.dz))]
    kz = np.abs(k[2][:nz + 1])
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + kz ** 2
    k2[0, 0, 0] = 1.0
    box = (2 * nx, 2 * ny, 2 * nz)
    rho = p.n_atoms * np.abs(psi) ** 2
    want = np.fft.irfftn(np.fft.rfftn(rho, box, axes=(0, 1, 2)) * (kz ** 2 / k2), box, axes=(0, 1, 2))[:nx, :ny, :nz]
    q = [2 * np.pi * np.fft.fftfreq(m, d) for m, d in zip(dims, (p.dx, p.dy, p.dz))]
    q2 = q[0][:, None, None] ** 2 + q[1][None, :, None] ** 2 + q[2] ** 2
    kin = np.fft.ifftn(np.fft.fftn(psi) * np.exp(-1j * p.real_time_dt / (2 * p.m) * q2))
    tol = 1e-13 if prec == "c128" else 1e-6
    # phi against the scale of the density it comes from
    assert np.linalg.norm(phi - want) < tol * np.linalg.norm(rho)
    assert rel_l2(out, kin) < tol
    assert abs(n - 1.0) < tol
