"""A chunk's frequencies run in up to three groups beside each other: a point's FP64 charge
and field are the same bits whatever its group and the number of points beside it (every
sum has a fixed order; the scaling comes from the highest frequency, which all sweeps
here share)."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('name,size', [('me0_16x64', (8, 13)), ('me1_64x256', (24, 50))])
def test_charges_do_not_depend_on_the_groups(built_lib, name, size):
    c = cases.make_case(name, seed=5, cols=size[0], rows=size[1], points=11)
    w = 2 * np.pi * c.freqs
    e = cases.engine_for(c)
    try:
        Q, st, _ = e.charges(w, 1.0, 'fp64')
        assert (st == 0).all()
        for n in (1, 2, 3, 4, 5, 7):
            Qn, st, _ = e.charges(w[-n:], 1.0, 'fp64')
            assert (st == 0).all()
            assert (Qn == Q[-n:]).all()
    finally:
        e.close()
