"""Symmetric systems whose leading pivot blocks are singular or nearly so: the symmetric
path searches pivots inside a block of at most 64 rows, so their points have to be solved
on the general path.  Dense 130-row systems (one front, blocks of 44 pivots in the order of
the DOFs): with the pivots of the whole front the error is that of test_gpu_pivot_blocks
(1e-16 x a condition and a growth of 1e3 each, times ten)."""
import numpy as np
import pytest
import scipy.sparse as sp

from sawsim_b200 import cases
from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu
N, BLOCK, W = 130, 44, 0.7


def _system(leading, seed=5):
    """(K, M, A at W, the electrode's column) with the leading block as named."""
    rng = np.random.default_rng(seed)
    m = N + 2
    A = rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))
    A = A + A.T
    U, s, _ = np.linalg.svd(A[:BLOCK, :BLOCK])
    if leading == 'zero':
        A[:BLOCK, :BLOCK] = 1e-300                   # in the pattern
    elif leading != 'regular':                       # Takagi-like: U diag(s) U^T is symmetric
        s[-1] = {'rank': 0.0, 'near': 1e-12}[leading]
        A[:BLOCK, :BLOCK] = (U * s) @ U.T
    M = np.diag(np.full(m, 0.1 + 0j))
    K = A + W * W * M
    return sp.csr_matrix(K), sp.csr_matrix(M), (K - W * W * M)[:N, :N], (K - W * W * M)[:N, N]


def _engine(K, M):
    return FrequencySolver.from_matrices(K, M, np.zeros(0, np.int64), np.array([N]), np.array([N + 1]), [])


@pytest.mark.parametrize('leading', ['regular', 'near', 'rank', 'zero'])
def test_leading_block(built_lib, leading):
    K, M, A, col = _system(leading)
    x = np.linalg.solve(A, -col)
    kq = K.toarray()[N, :N]
    lam = np.linalg.solve(A.T, kq)
    e = _engine(K, M)
    try:
        for _ in range(2):                           # the second call may go there directly
            disp, _, _ = e.solve(W)
            assert np.linalg.norm(disp[:N] - x) < 1e-9 * np.linalg.norm(x)
        s = e.stats()
        assert s['symmetric'] == float(leading == 'regular')
        assert np.linalg.norm(e.solve_adjoint(W, 'fp64') - lam) < 1e-9 * np.linalg.norm(lam)
        K2, M2, A2, col2 = _system('regular', 6)     # new values: the symmetric path again
        e.update_matrices(K2, M2)
        disp, _, _ = e.solve(W)
        x2 = np.linalg.solve(A2, -col2)
        assert np.linalg.norm(disp[:N] - x2) < 1e-9 * np.linalg.norm(x2)
        s = e.stats()
        assert s['symmetric'] == 1.0 and s['general_resolved'] == 0.0
    finally:
        e.close()


@pytest.mark.parametrize('fallback', [0, 1])
@pytest.mark.parametrize('precision', ['fp64', 'mixed', 'auto'])
@pytest.mark.parametrize('leading', ['regular', 'near', 'zero'])
def test_sweep_over_a_singular_leading_block(built_lib, leading, precision, fallback):
    """The leading block is singular at the middle frequency only (near, zero: M makes it
    regular at the others); every point has to be solved, in every precision."""
    K, M, _, _ = _system(leading)
    w = W * np.array([0.2, 0.6, 1.0, 1.0, 1.3])
    Kd, Md = K.toarray(), M.toarray()
    Q0 = []
    for wi in w:
        A = Kd - wi * wi * Md
        d = np.concatenate([np.linalg.solve(A[:N, :N], -A[:N, N]), [1.0, 0.0]])
        Q0.append(Kd[N] @ d)
    e = _engine(K, M)
    try:
        e.set_option('fp64_fallback', fallback)
        Q, st, _ = e.charges(w, 1.0, precision)
        assert (st == 0).all()
        # charges: sums of 130 products of entries of size 1 and a field with the error above
        assert np.max(np.abs(Q - Q0) / np.abs(Q0)) < (1e-8 if precision == 'fp64' else 1e-6)
    finally:
        e.close()


@pytest.mark.parametrize('kind', ['me0', 'me1', 'hex'])
def test_cells_do_not_need_it(built_lib, kind):
    c = (cases.make_hex_case('hex_8x4x48', seed=2, nx=8, ny=2, nz=13, points=9) if kind == 'hex' else
         cases.make_case('me0_16x64' if kind == 'me0' else 'me1_64x256', seed=2, cols=16, rows=64, points=9))
    e = cases.hex_engine_for(c) if kind == 'hex' else cases.engine_for(c)
    try:
        _, st, _ = e.charges(2 * np.pi * c.freqs, 1.0, 'fp64')
        s = e.stats()
    finally:
        e.close()
    assert (st == 0).all() and s['symmetric'] == 1.0 and s['general_resolved'] == 0.0
