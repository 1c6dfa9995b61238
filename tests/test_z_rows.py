"""The four-kernel schedule's z rows from nz = 16 on (nz = 8: the short runs against the
oracle at 64 x 32 x 8 in test_gpu_parity.py; this run's state collapses to a point there), and the dipolar lines of nx = 256 as two transforms at both tile widths,
against the split schedule in complex64.

Tolerance: 1e-5, thirty times the few 1e-7 that either schedule is off FP64 after these
iterations on this well-conditioned run."""
import numpy as np
import pytest

import gpesolver_b200 as G
from .helpers import gparams, rel_l2
from .test_gpu_parity import WELL_CONDITIONED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,tiles", [((64, 96, 16), None), ((32, 64, 24), None), ((32, 96, 32), None),
                                        ((32, 256, 64), None), ((256, 128, 24), "8,8"),
                                        ((256, 128, 32), "16,16"), ((256, 32, 16), "16,8")])
def test_z_rows_and_split_lines_match_split_schedule(dims, tiles, monkeypatch):
    if tiles:
        monkeypatch.setenv("GPE_X_TILES", tiles)
    p = gparams(WELL_CONDITIONED(*dims))
    out = []
    for sched in ("auto", "split"):
        with G.B200GrossPitaevskiSolver(p, precision="c64", schedule=sched) as s:
            s.load_pote(G.potential(p))
            s.load_buffer(G.initial_psi(p))
            s.imag_steps(12)
            a = s.export_data()
            s.real_steps(1, 0)
            s.real_steps(8, 1)
            out.append((a, s.export_data(), s.export_fi3d()))
    for a, b in zip(*out):
        assert rel_l2(a, b) < 1e-5
