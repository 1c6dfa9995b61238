"""A state that was loaded at any scale has the dipolar field of the normalised one, in the
passes with run-time line lengths and complex64, and so have its first imaginary-time steps.
The boundary is zero, as every initialiser leaves it: imaginary time keeps a boundary at the values
that were loaded (cpu_solver.cpp:50-97), so a non-zero one does depend on the scale.

Tolerance 2e-6: loading rounds psi at its own scale (6e-8 a component, 1e-7 in the density, sums
over the box average it), and the transforms round a stage at a time (1e-6, test_general_lines.py)."""
import numpy as np
import pytest

import gpesolver_b200 as G
from oracle import oracle as O

from .helpers import gparams, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-17, 1e-6, 3.0, 1e11, 1e13, 1e15, 1e17])
def test_field_and_first_steps_do_not_depend_on_the_loaded_scale(scale):
    dims = (10, 12, 9)
    p = gparams(O.default_config(nx=dims[0], ny=dims[1], nz=dims[2]))
    rng = np.random.default_rng(0)
    psi = rng.normal(size=dims) + 1j * rng.normal(size=dims)
    psi[[0, -1]] = psi[:, [0, -1]] = psi[:, :, [0, -1]] = 0
    out = []
    for f in (1.0, scale):
        with G.B200GrossPitaevskiSolver(p, precision="c64", schedule="split") as s:
            s.load_buffer(psi * f)
            s.calc_fi3d()
            phi = s.export_fi3d()
            s.imag_steps(1)
            phi1 = s.export_fi3d()
            s.imag_steps(2)
            out.append((phi, phi1, s.export_fi3d(), s.export_data()))
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        assert rel_l2(b, a) < 2e-6
