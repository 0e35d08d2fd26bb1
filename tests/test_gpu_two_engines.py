"""Two engines in one process: the kernels' shared-memory limits belong to the process, so an
engine of small fronts that runs in between must not lower them for one of large fronts
(another number of points makes the large engine launch and capture again)."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('symmetric', [0, 1])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_a_small_engine_beside_a_large_one(built_lib, precision, symmetric, monkeypatch):
    monkeypatch.setenv('SS_SYMMETRIC', str(symmetric))
    large = cases.make_hex_case('hex_8x4x48', seed=5, nx=8, ny=4, nz=14, points=5)       # 1,500 rows
    small = cases.make_case('me0_16x64', seed=5, cols=8, rows=13, points=3)
    w, ws = 2 * np.pi * large.freqs, 2 * np.pi * small.freqs
    e, f = cases.hex_engine_for(large), cases.engine_for(small)
    try:
        Q, st, _ = e.charges(w, 1.0, precision)
        assert (st == 0).all()
        assert (f.charges(ws, 1.0, precision)[1] == 0).all()
        Q1, st, _ = e.charges(w[-2:], 1.0, precision)
        assert (st == 0).all() and np.max(np.abs(Q1 - Q[-2:]) / np.abs(Q1)) < 1e-6
        lam = e.solve_adjoint(w[-1], 'fp64')
        assert np.isfinite(lam).all() and np.abs(lam).max() > 0
    finally:
        e.close()
        f.close()
