"""Products and reductions of the Krylov loop at the edges of their blocks: one warp per
row with eight frequencies a block, eight CTAs per frequency in the reductions.  Each
mixed-precision charge has to agree with the FP64 sweep of the same points to the 1e-6 of
the other mixed comparisons, whatever the number of points beside it."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('points', [1, 7, 8, 9, 17])
@pytest.mark.parametrize('name,size', [('me0_16x64', (8, 13)), ('me1_64x256', (8, 17))])
def test_mixed_charges_at_any_point_count(built_lib, name, size, points):
    c = cases.make_case(name, seed=5, cols=size[0], rows=size[1], points=18)
    w = 2 * np.pi * c.freqs[:points]
    e = cases.engine_for(c)
    try:
        Q, st, _ = e.charges(w, 1.0, 'mixed')
        assert (st == 0).all()
        Q0, st0, _ = e.charges(w, 1.0, 'fp64')
        assert (st0 == 0).all()
    finally:
        e.close()
    assert np.max(np.abs(Q - Q0) / np.abs(Q0)) < 1e-6
