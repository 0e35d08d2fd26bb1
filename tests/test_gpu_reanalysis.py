"""Another boundary condition on an engine that has solved an adjoint: the transposed pattern
belongs to the analysis, so the adjoint has to equal a fresh engine's bit for bit (every
sum has a fixed order; the general path's tiles are forced, since its tuner may pick others
for another engine).  The boundary sets differ in size and in which DOFs they hold."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('symmetric', [0, 1])
def test_adjoint_after_another_boundary_condition(built_lib, symmetric, monkeypatch):
    monkeypatch.setenv('SS_SYMMETRIC', str(symmetric))
    if not symmetric:
        monkeypatch.setenv('SS_SCHUR_TILE', '2')
    c = cases.make_case('me1_64x256', seed=5, cols=8, rows=17, points=3)
    w = 2 * np.pi * c.freqs[1]
    fix, plus, minus, groups = c.bc[:4]
    rest = np.setdiff1d(np.arange(2 * c.mesh.N), np.concatenate([np.ravel(v) for v in (fix, plus, minus)] +
                                                                 [np.ravel(g) for g in groups]))
    more = np.concatenate([np.ravel(fix), rest[::37]])
    e, fresh = cases.engine_for(c), cases.engine_for(c)
    try:
        fresh._set_bc((more, plus, minus, groups))
        want = fresh.solve_adjoint(w, 'fp64')
        first = e.solve_adjoint(w, 'fp64')
        e._set_bc((more, plus, minus, groups))
        assert np.array_equal(e.solve_adjoint(w, 'fp64'), want)
        e._set_bc((fix, plus, minus, groups))
        assert np.array_equal(e.solve_adjoint(w, 'fp64'), first)
    finally:
        e.close()
        fresh.close()
