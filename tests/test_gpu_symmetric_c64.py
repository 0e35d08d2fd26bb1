"""Mixed sweeps on the symmetric path with nothing to fall back on: each complex64 update
candidate forced in turn (the TMA tiles of 128 and 64 columns, the SIMT tiles), on fronts of
one to eight pivot blocks and up to two groups of them (updates from two children, in place,
inside a group and past it, with remainder tiles).  A wrong tile makes factors that are
wrong in the first digit: the points then do not converge, or take many Krylov steps.  Sound
complex64 factors of the two paths have backward errors of the same order, so the steps per
point may differ by one."""
import numpy as np
import pytest

from sawsim_b200 import _lib as L, cases
from sawsim_b200.engine import FrequencySolver

pytestmark = pytest.mark.gpu

CELLS = [('hex', (8, 1, 6)), ('hex', (8, 2, 13)), ('hex', (8, 3, 9)), ('hex', (8, 4, 10)), ('me0_16x64', (8, 13)),
         ('me0_16x64', (16, 41)), ('me1_64x256', (24, 50)), ('me1_64x256', (40, 44))]


def _engine(kind, size, points=4):
    if kind == 'hex':
        c = cases.make_hex_case('hex_8x4x48', seed=3, nx=size[0], ny=size[1], nz=size[2], points=points)
        return c, cases.hex_engine_for(c)
    c = cases.make_case(kind, seed=3, cols=size[0], rows=size[1], points=points)
    return c, cases.engine_for(c)


def _mixed(kind, size):
    c, e = _engine(kind, size)
    w = 2 * np.pi * c.freqs
    try:
        e.set_option('fp64_fallback', 0)
        Q, st, _ = e.charges(w, 1.0, 'mixed')
        s = e.stats()
        assert (st == 0).all() and s['fp64_resolved'] == s['general_resolved'] == s['mixed_not_converged'] == 0.0
        Q0, st0, _ = e.charges(w, 1.0, 'fp64')
        assert (st0 == 0).all()
    finally:
        e.close()
    assert np.max(np.abs(Q - Q0) / np.abs(Q0)) < 1e-6
    return s


@pytest.mark.parametrize('kind,size', CELLS)
@pytest.mark.parametrize('tile', [None, 0, 1, 2])
def test_update_candidates(built_lib, kind, size, tile, monkeypatch):
    monkeypatch.setenv('SS_SYMMETRIC', '0')
    steps = _mixed(kind, size)['krylov_steps_primal']
    monkeypatch.delenv('SS_SYMMETRIC')
    if tile is not None:
        monkeypatch.setenv('SS_SYM_TILE_C64', str(tile))
    s = _mixed(kind, size)
    assert s['symmetric'] == 1.0 and s['krylov_steps_primal'] <= steps + 4
    if tile is not None and kind == 'hex':
        assert s[f'schur_candidate{tile}'] > 0.0


@pytest.mark.parametrize('points', [1, 7, 8, 9, 17])
@pytest.mark.parametrize('name,size', [('me0_16x64', (8, 13)), ('me1_64x256', (8, 17))])
def test_krylov_loop_at_any_point_count(built_lib, name, size, points):
    """The Krylov loop's blocks of eight frequencies: these cells converge in a step or two."""
    c, e = _engine(name, size, points=18)
    w = 2 * np.pi * c.freqs[:points]
    try:
        e.set_option('fp64_fallback', 0)
        Q, st, _ = e.charges(w, 1.0, 'mixed')
        s = e.stats()
        Q0, st0, _ = e.charges(w, 1.0, 'fp64')
    finally:
        e.close()
    assert (st == 0).all() and (st0 == 0).all() and s['general_resolved'] == 0.0
    assert s['krylov_steps_primal'] <= 2 * points
    assert np.max(np.abs(Q - Q0) / np.abs(Q0)) < 1e-6


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_mesh_and_matrix_engines_agree_bit_for_bit(built_lib, precision, monkeypatch):
    """The symmetric path of a mesh engine and of its exported matrices on the same nodes."""
    monkeypatch.setenv('SS_SYM_TILE_C64', '0')           # one candidate in both
    c, g = _engine('me1_64x256', (16, 37))
    node = np.tile(np.arange(c.mesh.N), 4)
    try:
        K, M = g.export(L.SS_MAT_K), g.export(L.SS_MAT_M)
        e = FrequencySolver.from_matrices(K, M, *c.bc, dof_node=node, node_xyz=c.mesh.pos_m[:, :2])
        try:
            w = 2 * np.pi * c.freqs
            Qg, _, _ = g.charges(w, 1.0, precision)
            Qe, st, _ = e.charges(w, 1.0, precision)
            assert (st == 0).all() and e.stats()['symmetric'] == g.stats()['symmetric'] == 1.0
            assert np.array_equal(Qg, Qe)
        finally:
            e.close()
    finally:
        g.close()
