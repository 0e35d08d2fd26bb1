"""Sweeps whose graphs have different numbers of frequency groups on one engine (one and two
points run in one and two groups, more in three): the timed updates counted are those of
the graph that ran, and a sweep of several chunks whose last one is short returns what the
same points return beside others."""
import numpy as np
import pytest

from sawsim_b200 import cases

pytestmark = pytest.mark.gpu


def test_update_times_belong_to_the_sweep(built_lib):
    """The first points' update time, a one-point sweep, the first points again: a count kept
    from the other graph reads a third of the pairs, or three times as many."""
    c = cases.make_case('me1_64x256', seed=5, cols=16, rows=41, points=11)
    w = 2 * np.pi * c.freqs
    e = cases.engine_for(c)

    def updates(points):
        ms = []
        for _ in range(4):                       # the first one captures
            e.charges(points, 1.0, 'fp64')
            ms.append(e.stats()['schur_gemm_ms'])
        return np.array(ms[1:])
    try:
        one = updates(w[-1:])
        wide = updates(w)
        one2 = updates(w[-1:])
        wide2 = updates(w)
    finally:
        e.close()
    assert wide2.min() > 0.6 * wide.min()
    assert one2.min() < one.min() + 0.3 * wide.min()


@pytest.mark.parametrize('last', [1, 2, 3])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_short_last_chunk(built_lib, last, precision):
    """256 points a chunk; the scaling comes from the highest frequency, which all these
    sweeps share, so the FP64 charges are equal bit for bit (the mixed ones to 1e-6, the bar of
    the other mixed comparisons: their Krylov steps stop with the chunk's last point)."""
    c = cases.make_case('me0_16x64', seed=5, cols=8, rows=13, points=256 + last)
    w = 2 * np.pi * c.freqs
    e = cases.engine_for(c)
    try:
        e.set_option('fp64_fallback', 0)
        for _ in range(2):
            Q, st, _ = e.charges(w, 1.0, precision)
            s = e.stats()
            assert (st == 0).all() and s['symmetric'] == 1.0 and s['chunk'] == 256
        Q1, st, _ = e.charges(w[last:], 1.0, precision)
        assert (st == 0).all()
        Q2, st, _ = e.charges(w[-5:], 1.0, precision)
        assert (st == 0).all()
    finally:
        e.close()
    if precision == 'fp64':
        assert (Q1 == Q[last:]).all() and (Q2 == Q[-5:]).all()
    else:
        assert np.max(np.abs(Q1 - Q[last:]) / np.abs(Q1)) < 1e-6 and np.max(np.abs(Q2 - Q[-5:]) / np.abs(Q2)) < 1e-6
