"""Matrices that are symmetric to a few units in the 14th digit, inside or in the electrode's
row and column: the symmetric path may factor them, but their adjoint has to be the transposed
system's, not the primal solution.  Condition of the 60 x 60
systems below 10, products of 60 terms: a refined solution is right to some 10 x 1.1e-16 x
sqrt(60) = 1e-14; the asymmetry, taken for none, would leave several times that."""
import numpy as np
import pytest
import scipy.sparse as sp

from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu
N, W = 60, 0.7


@pytest.mark.parametrize('where', ['nowhere', 'inside', 'electrode'])
def test_adjoint_of_a_nearly_symmetric_system(built_lib, where):
    rng = np.random.default_rng(7)
    A = rng.standard_normal((N + 2, N + 2)) + 1j * rng.standard_normal((N + 2, N + 2))
    A = (A + A.T) / 40 + (2 + 0.3j) * np.eye(N + 2)
    if where == 'inside':
        A[:N, :N] += np.tril(rng.choice([-1, 1], (N, N)) * 9e-14, -1)
    if where == 'electrode':
        A[:N, N] *= 1 + rng.choice([-1, 1], N) * 9e-14
    M = np.eye(N + 2) * (0.1 + 0j)
    K = A + W * W * M
    A = K - W * W * M
    assert np.linalg.cond(A[:N, :N]) < 10
    x = np.linalg.solve(A[:N, :N], -A[:N, N])
    lam = np.linalg.solve(A[:N, :N].T, K[N, :N])
    e = FrequencySolver.from_matrices(sp.csr_matrix(K), sp.csr_matrix(M), np.zeros(0, np.int64), np.array([N]),
                                      np.array([N + 1]), [])
    try:
        disp, _, _ = e.solve(W)
        assert e.stats()['symmetric'] == 1.0
        assert np.linalg.norm(disp[:N] - x) < 1e-14 * np.linalg.norm(x)
        assert np.linalg.norm(e.solve_adjoint(W, 'fp64') - lam) < 1e-14 * np.linalg.norm(lam)
    finally:
        e.close()
