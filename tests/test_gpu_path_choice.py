"""Which path an engine takes follows its values: a system found unsymmetric keeps to the
general path at other top frequencies too, and takes the symmetric one when its values
become symmetric again.  The charges are those of a fresh engine: on the symmetric path bit for
bit, on the general one, whose tuner may pick other tiles for another engine, to 1e-7 (the
bar of the oracle comparisons)."""
import numpy as np
import pytest

from sawsim_b200 import _lib as L, cases
from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu


def test_the_path_follows_the_values(built_lib):
    c = cases.make_case('me1_64x256', seed=3, cols=8, rows=16, points=4)
    g = cases.engine_for(c)
    K, M = g.export(L.SS_MAT_K), g.export(L.SS_MAT_M)
    g.close()
    U = K.copy()
    row = np.repeat(np.arange(U.shape[0]), np.diff(U.indptr))
    U.data[(row >= 200) & (row < 400) & (U.indices > row)] *= 1.001
    w = 2 * np.pi * c.freqs

    def charges(e, symmetric):
        out = []
        for n in (4, 2, 4):                          # two top frequencies, the first one again
            Q, st, _ = e.charges(w[:n], 1.0, 'fp64')
            assert (st == 0).all() and e.stats()['symmetric'] == float(symmetric)
            out.append(Q)
        return np.concatenate(out)

    fresh = {}
    for name, A in (('U', U), ('K', K)):
        f = FrequencySolver.from_matrices(A, M, *c.bc)
        fresh[name] = charges(f, name == 'K')
        f.close()
    e = FrequencySolver.from_matrices(U, M, *c.bc)
    try:
        assert np.max(np.abs(charges(e, False) - fresh['U']) / np.abs(fresh['U'])) < 1e-7
        e.update_matrices(K, M)
        assert np.array_equal(charges(e, True), fresh['K'])
        e.update_matrices(U, M)
        assert np.max(np.abs(charges(e, False) - fresh['U']) / np.abs(fresh['U'])) < 1e-7
    finally:
        e.close()
