"""The reciprocal of a pivot, seen without the refinement that would hide it: one front of
DOFs without coupling, so that the direct solve of each is b times the reciprocal of its
pivot.  Its relative residual, which the library prints with SS_DEBUG_IR, has to stay below
six roundings: |z|^2 (at most two of them), its reciprocal (one), the product with conj(z) (one),
the product with b (two), 6 x 1.1e-16 = 6.7e-16."""
import re

import numpy as np
import pytest
import scipy.sparse as sp

from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 16, 17, 33, 64])
def test_direct_solve_of_uncoupled_dofs(built_lib, n, monkeypatch, capfd):
    rng = np.random.default_rng(n)
    # mantissas and phases over their whole ranges; the equilibration takes the powers of two out
    a = rng.uniform(1, 4, n) * 2.0 ** rng.integers(-20, 20, n) * np.exp(2j * np.pi * rng.random(n))
    K = sp.lil_matrix((n + 2, n + 2), dtype=complex)
    K.setdiag(np.concatenate([a, [1, 1]]))
    K[:n, n] = (a * rng.uniform(0.5, 2, n))[:, None]
    K[n, :n] = K[:n, n].T
    M = sp.csr_matrix(sp.identity(n + 2) * (1e-30 + 0j))
    node = np.concatenate([np.zeros(n, np.int64), [1, 2]])
    monkeypatch.setenv('SS_DEBUG_IR', '1')
    e = FrequencySolver.from_matrices(sp.csr_matrix(K), M, np.zeros(0, np.int64), np.array([n]), np.array([n + 1]), [],
                                      dof_node=node)
    try:
        e.solve(1.0)
        assert e.stats()['symmetric'] == 1.0
    finally:
        e.close()
    res = re.findall(r'direct solve \(c128\): \|r\|/\|b\| f0 (\S+)', capfd.readouterr().err)
    assert len(res) == 1 and float(res[0]) < 6.7e-16
