"""Fronts merged with their only child (host analysis, CPU): no mergeable pair is
left, and the trees stay valid with exact fill on slabs whose dissection makes such
chains and on a 2D cell that has none."""
import numpy as np
import pytest

from test_analysis import _check_fill, _check_tree, _hex, _q9
from sawsim_b200.analysis import analyze_hex27, analyze_q9

MERGE_PIVOTS = 256


@pytest.mark.parametrize('cell', [('hex', 8, 1, 6), ('hex', 8, 3, 7), ('me1_64x256', 16, 21)])
def test_only_children_are_merged(cell):
    if cell[0] == 'hex':
        c, T, active, S = _hex(*cell[1:])
        a = analyze_hex27(c.pos_m, c.hexas, c.bc)
    else:
        c, bc, T, active, S = _q9(*cell)
        a = analyze_q9(c.mesh.pos_m, c.mesh.quads, bc)
    _check_tree(a)
    _check_fill(a, T, active, S)
    kids = np.bincount(a.parent[a.parent >= 0], minlength=a.k.size)
    for f in np.flatnonzero(a.parent >= 0):
        p = a.parent[f]
        if kids[p] == 1 and a.m[f] - a.k[f] == a.m[p]:
            assert a.k[f] + a.k[p] > MERGE_PIVOTS
