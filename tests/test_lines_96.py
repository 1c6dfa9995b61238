"""The compiled transforms of lengths 24, 48, 96 and 192 (grids with 96 and 24: second
stages of radix 6 and 12) on every axis and in every kernel that runs them, against the
split schedule: one imaginary- and one real-time stretch in complex64.

Tolerance: 1e-5, thirty times the few 1e-7 that either schedule is off FP64 after these
iterations on this well-conditioned run."""
import numpy as np
import pytest

import gpesolver_b200 as G
from .helpers import gparams, rel_l2
from .test_gpu_parity import WELL_CONDITIONED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("dims", [(96, 96, 24), (96, 32, 16), (32, 96, 24), (96, 128, 24), (64, 96, 8), (32, 64, 24)])
def test_96_matches_split(dims, pair, monkeypatch):
    monkeypatch.setenv("GPE_PLANE_PAIR", pair)
    p = gparams(WELL_CONDITIONED(*dims))
    out = []
    for sched in ("auto", "split"):
        with G.B200GrossPitaevskiSolver(p, precision="c64", schedule=sched) as s:
            s.load_pote(G.potential(p))
            s.load_buffer(G.initial_psi(p))
            s.imag_steps(20)
            s.real_steps(10, 0)
            out.append((s.export_data(), s.export_fi3d()))
    for a, b in zip(*out):
        assert rel_l2(a, b) < 1e-5
