"""Reassembly on an analysed engine: the mesh's gather lists are kept on the device and
the element matrices are formed in the front arena of the sweep before.  K and M are
fixed-order sums, so they have to equal a fresh engine's bit for bit."""
import numpy as np
import pytest

from sawsim_b200 import _lib as L, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['me0', 'me1', 'hex'])
def test_reassembled_matrices_equal_a_fresh_engines(built_lib, kind):
    if kind == 'hex':
        c = cases.make_hex_case('hex_8x4x48', seed=2, nx=8, ny=1, nz=7, points=3)
        make = cases.hex_engine_for
    else:
        c = cases.make_case('me0_16x64' if kind == 'me0' else 'me1_64x256', seed=2, cols=8, rows=15, points=3)
        make = cases.engine_for
    w = 2 * np.pi * c.freqs
    top = 0.9 * c.omega_top
    e, fresh = make(c), make(c)
    try:
        Q0, _, _ = e.charges(w, 1.0, 'fp64')
        e.set_freeze_frequency(top)
        fresh.set_freeze_frequency(top)
        for which in (L.SS_MAT_K, L.SS_MAT_M):
            a, b = e.export(which), fresh.export(which)
            assert np.array_equal(a.indices, b.indices) and np.array_equal(a.data, b.data)
        Q1, _, _ = e.charges(w, 1.0, 'fp64')
        assert np.array_equal(Q1, fresh.charges(w, 1.0, 'fp64')[0]) and not np.array_equal(Q0, Q1)
        e.set_freeze_frequency(c.omega_top)
        assert np.array_equal(e.charges(w, 1.0, 'fp64')[0], Q0)
    finally:
        e.close()
        fresh.close()
