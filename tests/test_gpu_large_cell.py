"""A cell of 1,049,608 DOF, whose condition of some 1e11 lets the symmetric factors miss its
nearly singular mode: the charges have to agree with the general path's to 1e-8 (both are
refined to better than 1e-9), and the fields, which hold that mode, to the condition times the
unit roundoff and the general factors' own growth, 1e-2."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


def test_charges_and_fields_of_a_large_cell(built_lib, monkeypatch):
    c = cases.make_case('me1_64x256', seed=0, cols=128, rows=512, points=9)
    w = 2 * np.pi * c.freqs
    e = cases.engine_for(c)
    try:
        Q, st, _ = e.charges(w, 1.0, 'fp64')
        assert (st == 0).all()
        d, q, _ = e.solve(w[-1])
        Qr, _, _ = e.charges(w, 1.0, 'fp64')
        monkeypatch.setenv('SS_SYMMETRIC', '0')
        Q0, st0, _ = e.charges(w, 1.0, 'fp64')
        d0, _, _ = e.solve(w[-1])
        assert (st0 == 0).all() and e.stats()['symmetric'] == 0.0
    finally:
        e.close()
    assert np.max(np.abs(Q - Q0) / np.abs(Q0)) < 1e-8 and np.max(np.abs(Qr - Q0) / np.abs(Q0)) < 1e-8
    assert abs(q - Q0[-1]) < 1e-8 * abs(Q0[-1])
    assert np.linalg.norm(d - d0) < 1e-2 * np.linalg.norm(d0)
