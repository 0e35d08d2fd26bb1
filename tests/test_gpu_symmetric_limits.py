"""Fronts at the limit of the symmetric solve kernels' shared memory: they hold a block of
64 x 65 entries and a front's vector, so a complex128 front of more than 10,368 rows has to
take the general path (whose solves hold a 32 x 32 block).  Tridiagonal systems whose DOFs
share a node, so that they are one dense front; condition below 10."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import spsolve

from sawsim_b200.analysis import analyze_csr
from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu
W = 0.7


def _chain(n):
    """n DOFs of one node in a chain, and the electrodes, + joined to the first DOF."""
    off = np.full(n + 1, -1 + 0.1j)
    off[n - 1:] = 0.0                            # the electrodes are not part of the chain
    A = sp.diags([off, np.full(n + 2, 4 + 0.2j), off], [-1, 0, 1]).tolil()
    A[0, n] = A[n, 0] = 0.5
    A = sp.csr_matrix(A)
    A.eliminate_zeros()
    M = sp.csr_matrix(sp.identity(n + 2) * (0.1 + 0j))
    node = np.concatenate([np.zeros(n, np.int64), [1, 2]])
    return A, M, node, (np.zeros(0, np.int64), np.array([n]), np.array([n + 1]), [])


@pytest.mark.parametrize('n,symmetric', [(10360, True), (10400, False)])
def test_front_at_the_limit(built_lib, n, symmetric):
    K, M, node, bc = _chain(n)
    assert analyze_csr(K, bc, dof_node=node).max_front == n
    e = FrequencySolver.from_matrices(K, M, *bc, dof_node=node)
    try:
        disp, _, _ = e.solve(W)
        assert e.stats()['symmetric'] == float(symmetric)
    finally:
        e.close()
    A = sp.csc_matrix(K - W * W * M)
    x = spsolve(A[:n, :n], -A[:n, n].toarray().ravel())
    assert np.linalg.norm(disp[:n] - x) < 1e-12 * np.linalg.norm(x)
