"""gpe_time_kernel's byte count of the z rows (four-kernel schedule): what the timed mode, a middle
real-time iteration, moves."""
import ctypes

import numpy as np
import pytest

import gpesolver_b200 as G
from gpesolver_b200 import capi
from oracle import oracle as O

from .helpers import gparams

pytestmark = pytest.mark.gpu

GPE_K_F_Z = 14


def test_z_rows_count_no_phi_store():
    dims = (64, 32, 8)
    n = dims[0] * dims[1] * dims[2]
    p = gparams(O.default_config(nx=dims[0], ny=dims[1], nz=dims[2]))
    assert capi.lib().gpe_kernel_name(GPE_K_F_Z) == b"k2_z"
    ms, b = ctypes.c_double(), ctypes.c_double()
    with G.B200GrossPitaevskiSolver(p) as s:
        s.load_buffer(np.ones(dims, dtype=np.complex128))
        capi.check(capi.lib().gpe_time_kernel(s.handle, GPE_K_F_Z, 2, ctypes.byref(ms), ctypes.byref(b)))
    # increment and psi in and out, ny of 2 ny spectrum rows in and out (8 bytes each), V in (4)
    assert b.value == n * (4 * 8 + 2 * 8 + 4)
