"""The symmetric path of the factorisation (fronts of a complex symmetric scaled
system: upper update blocks, gathered children, narrow and wide fronts) against the
general path on the same engine inputs, and the systems that must keep the general
path.  Both paths solve the same equilibrated system to a normwise backward error
near the unit roundoff, so the FP64 charges agree to the conditioning of these cells
(1e-7 relative, the bar of the oracle comparisons; the mixed ones to 1e-6) and the
fields have backward errors below 1e-12 in the oracle's own system."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import oracle_engine
from sawsim_b200 import _lib as L, cases
from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu


def _build(kind, size):
    if kind == 'hex':
        c = cases.make_hex_case('hex_8x4x48', seed=3, nx=size[0], ny=size[1], nz=size[2], points=4)
        return c, lambda: cases.hex_engine_for(c)
    c = cases.make_case(kind, seed=3, cols=size[0], rows=size[1], points=4)
    return c, lambda: cases.engine_for(c)


def _charges(make, w, precision, monkeypatch, sym):
    monkeypatch.setenv('SS_SYMMETRIC', '1' if sym else '0')
    e = make()
    try:
        Q, st, _ = e.charges(w, 1.0, precision)
        lam = e.solve_adjoint(w[1], 'fp64') if precision == 'fp64' else None
        s = e.stats()
    finally:
        e.close()
    assert (st == 0).all() and s['symmetric'] == float(sym)
    return Q, lam


# sizes whose fronts end on and off the tiles: one pivot block up to two groups of
# blocks (k > 256), update blocks below and above one 64-wide tile
@pytest.mark.parametrize('kind,size', [('me0_16x64', (8, 13)), ('me0_16x64', (16, 41)), ('me1_64x256', (8, 16)),
                                       ('me1_64x256', (16, 37)), ('me1_64x256', (24, 50)), ('me1_64x256', (40, 44)),
                                       ('hex', (8, 1, 6)),
                                       ('hex', (8, 2, 13))])
@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_symmetric_path_equals_the_general_path(built_lib, kind, size, precision, monkeypatch):
    c, make = _build(kind, size)
    w = 2 * np.pi * c.freqs
    Q0, l0 = _charges(make, w, precision, monkeypatch, False)
    Q1, l1 = _charges(make, w, precision, monkeypatch, True)
    assert np.max(np.abs(Q1 - Q0) / np.abs(Q0)) < (1e-7 if precision == 'fp64' else 1e-6)
    if precision == 'fp64':
        assert np.linalg.norm(l1 - l0) / np.linalg.norm(l0) < 1e-6


@pytest.mark.parametrize('name,size', [('me1_64x256', (16, 37)), ('me0_16x64', (16, 41))])
def test_symmetric_fields_solve_the_oracle_system(built_lib, name, size):
    c = cases.make_case(name, seed=3, cols=size[0], rows=size[1], points=3)
    _, _, o = oracle_engine(c)
    e = cases.engine_for(c)
    try:
        for f in c.freqs:
            w = 2 * np.pi * f
            A, rhs = o.system(w)
            disp, _, _ = e.solve(w)
            x = disp[o.active]
            r = np.abs(rhs - A @ x)
            assert np.linalg.norm(r) / (sp.linalg.norm(A) * np.linalg.norm(x) + np.linalg.norm(rhs)) < 1e-12
        assert e.stats()['symmetric'] == 1.0
    finally:
        e.close()


@pytest.mark.parametrize('which', ['K', 'M'])
def test_a_matrix_that_is_not_symmetric_keeps_the_general_path(built_lib, which):
    """The assembled K or M made unsymmetric in some rows: the general path, and the
    oracle's charges for those matrices."""
    from oracle.solver import FrequencySolver as Oracle
    c = cases.make_case('me1_64x256', seed=3, cols=8, rows=16, points=3)
    g = cases.engine_for(c)
    K, M = g.export(L.SS_MAT_K), g.export(L.SS_MAT_M)
    g.close()
    A = K if which == 'K' else M
    row = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    A.data[(row >= 200) & (row < 400) & (A.indices > row)] *= 1.001
    w = 2 * np.pi * c.freqs
    e = FrequencySolver.from_matrices(K, M, *c.bc)
    try:
        Q, st, _ = e.charges(w, 1.0, 'fp64')
        assert (st == 0).all() and e.stats()['symmetric'] == 0.0
    finally:
        e.close()
    Qo = Oracle(K, M, *c.bc).sweep(c.freqs)
    assert np.max(np.abs(Q - Qo) / np.abs(Qo)) < 1e-7


def test_anisotropic_pml_slab_keeps_the_general_path(built_lib):
    """A Hex27 slab whose PML takes the rotated crystal: the Voigt stretch multipliers
    and the conjugated coupling make K unsymmetric, so the general path runs."""
    c = cases.make_hex_case('hex_8x4x48', seed=3, nx=8, ny=1, nz=6, points=3)
    c.mat_idx[c.cell.hex_tag == c.cell.pml_tag] = 0
    e = cases.hex_engine_for(c)
    try:
        e.charges(2 * np.pi * c.freqs, 1.0, 'fp64')
        assert e.stats()['symmetric'] == 0.0
    finally:
        e.close()


@pytest.mark.parametrize('kind,size', [('me0_16x64', (8, 13)), ('me1_64x256', (8, 17))])
@pytest.mark.parametrize('scale', [1.0, 1.5])
def test_adjoint_solutions_of_a_symmetric_system(built_lib, kind, size, scale):
    """The adjoint fields A^T l = kq, with the electrode's column proportional to its row
    (one solve serves both) and with half of it scaled (two solves), in the oracle's system:
    backward errors as for the fields."""
    from oracle.solver import FrequencySolver as Oracle
    c, make = _build(kind, size)
    g = make()
    K, M = g.export(L.SS_MAT_K), g.export(L.SS_MAT_M)
    g.close()
    zheng = np.asarray(c.bc[1], dtype=np.int64)
    row = np.repeat(np.arange(K.shape[0]), np.diff(K.indptr))
    K.data[np.isin(K.indices, zheng) & ~np.isin(row, zheng) & (row % 2 == 0)] *= scale
    o = Oracle(K, M, *c.bc)
    e = FrequencySolver.from_matrices(K, M, *c.bc)
    try:
        for f in c.freqs[:2]:
            w = 2 * np.pi * f
            A, _ = o.system(w)
            lam = e.solve_adjoint(w, 'fp64')
            Q, st, _ = e.charges(np.array([w]), 1.0, 'mixed')
            Q0, st0, _ = e.charges(np.array([w]), 1.0, 'fp64')
            kq = (o._T.T @ o.kts)[o.active]
            r = A.T @ lam - kq
            assert np.linalg.norm(r) / (sp.linalg.norm(A) * np.linalg.norm(lam) + np.linalg.norm(kq)) < 1e-12
            assert st[0] == 0 and st0[0] == 0 and abs(Q[0] - Q0[0]) < 1e-6 * abs(Q0[0])
        assert e.stats()['symmetric'] == 1.0
    finally:
        e.close()
