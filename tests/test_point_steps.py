"""The interface's pointwise steps alone (potential half step, Euler step) against numpy, where a
grid is smaller than a block, ragged, has long rows, or has more points than threads are resident.

Tolerances: complex128, 1e-14 of psi (three to ten roundings of 1e-16 on each point, terms of the
size of psi); complex64, 1e-6 likewise (6e-8 a rounding; psi and V are rounded on loading)."""
import numpy as np
import pytest

import gpesolver_b200 as G
from oracle import oracle as O

from .helpers import gparams, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("c128", 1e-14), ("c64", 1e-6)])
@pytest.mark.parametrize("dims", [(3, 3, 3), (1, 4, 5), (7, 5, 9), (4, 3, 1600), (640, 5, 4), (3, 700, 3), (96, 90, 50)])
def test_steps_match_numpy(dims, prec, tol):
    p = gparams(O.default_config(nx=dims[0], ny=dims[1], nz=dims[2]))
    rng = np.random.default_rng(sum(dims))
    psi = rng.normal(size=dims) + 1j * rng.normal(size=dims)
    psi /= np.sqrt((np.abs(psi) ** 2).sum() * p.dx * p.dy * p.dz)
    V = rng.uniform(0, 1, dims) / p.real_time_dt  # half a radian at most from V and from phi
    phi = rng.uniform(-1, 1, dims) / (p.real_time_dt * p.cdd)
    inside = np.zeros(dims, bool)
    inside[1:-1, 1:-1, 1:-1] = True
    with G.B200GrossPitaevskiSolver(p, precision=prec, schedule="split") as s:
        s.load_pote(V)
        s.import_data(psi)
        s.load_fi3d(phi)
        s.real_fft_potential_half_step()
        half = s.export_data()
        s.import_data(psi)
        s.imag_iter_linear_step()
        s.imag_iter_nonlinear_step()
        euler = s.export_data()
    dens = np.abs(psi) ** 2
    h = V + p.cdd * phi + (p.ggp11 - p.cdd / 3) * p.n_atoms * dens + p.gamma * p.w_15 * dens * np.sqrt(dens)
    want = np.where(inside, psi * np.exp(-0.5j * p.real_time_dt * h), psi)
    assert rel_l2(half, want) < tol
    want = h * psi
    for axis, (d, sign) in enumerate(((p.dx, 1.0), (p.dy, -1.0), (p.dz, -1.0))):
        # the x term's sign is the reference's (cpu_solver.cpp:59-67)
        lap = np.roll(psi, 1, axis) + np.roll(psi, -1, axis) - 2 * psi
        want = want + sign * (-0.5 if axis == 0 else 0.5) / (p.m * d * d) * lap
    want = np.where(inside, psi - p.imag_time_dt * want, psi)
    assert rel_l2(euler, want) < tol


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("dims", [(3, 3, 3), (1, 1, 1), (5, 7, 3), (4, 3, 1600), (300, 12, 8), (96, 90, 50), (384, 384, 9)])
def test_norm_matches_numpy(dims, prec):
    """Sums of squares in FP64 over parts of rows: 1e-13 from numpy's, on psi as the precision holds it; the
    last grid has several parts per CTA.  The same to the bit when asked again."""
    p = gparams(O.default_config(nx=dims[0], ny=dims[1], nz=dims[2]))
    rng = np.random.default_rng(sum(dims))
    psi = rng.normal(size=dims) + 1j * rng.normal(size=dims)
    if prec == "c64":
        psi = psi.astype(np.complex64).astype(np.complex128)
    with G.B200GrossPitaevskiSolver(p, precision=prec, schedule="split") as s:
        s.import_data(psi)
        got = [s.calc_norm() for _ in range(3)]
    want = (np.abs(psi) ** 2).sum() * p.dx * p.dy * p.dz
    assert abs(got[0] - want) < 1e-13 * want
    assert got[1:] == got[:1] * 2
