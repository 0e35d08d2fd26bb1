"""The LU of a pivot block at the edges of its layout (groups of four columns, 16 columns
and up to 64 rows per block): dense complex symmetric systems with a zero diagonal, so that
the pivots come from interchanges, against numpy in 64 bits.  A random matrix of these
sizes has a condition number of some 1e3 and a growth below 1e3, so the field after the
refinement step is right to 1e-16 x 1e6 = 1e-10; the bar is ten times that."""
import numpy as np
import pytest
import scipy.sparse as sp

from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 3, 4, 5, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 130])
def test_dense_symmetric_pivot_blocks(built_lib, n):
    rng = np.random.default_rng(n)
    m = n + 2                                # the two last DOFs: + and - electrode
    A = rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))
    A = A + A.T
    if n > 1:
        A[np.arange(m), np.arange(m)] = 1e-14        # in the pattern, useless as pivots
    K, M = sp.csr_matrix(A), sp.csr_matrix((np.full(m, 0.1 + 0j), (np.arange(m), np.arange(m))), shape=(m, m))
    e = FrequencySolver.from_matrices(K, M, np.zeros(0, np.int64), np.array([n]), np.array([n + 1]), [])
    try:
        w = 0.7
        disp, _, _ = e.solve(w)
    finally:
        e.close()
    B = A - w * w * M.toarray()
    x = np.linalg.solve(B[:n, :n], -B[:n, n])
    assert np.linalg.norm(disp[:n] - x) < 1e-9 * np.linalg.norm(x)
