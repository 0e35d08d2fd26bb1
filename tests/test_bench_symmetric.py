"""bench.py's roofline entries and the statistics behind them on the symmetric path: they
describe the kernels that ran there, and the general path's slots read 0 or what the
header says."""
from types import SimpleNamespace

import numpy as np
import pytest

from test_bench_contract import _FakeEngine, bench   # noqa: F401
from sawsim_b200 import cases


@pytest.mark.parametrize('used', ['fp64', 'mixed'])
def test_rooflines_describe_the_symmetric_factorisation(bench, used):   # noqa: F811
    c = SimpleNamespace(name='me1_64x256', mesh=SimpleNamespace(ne=2, N=6))
    s = dict(symmetric=1.0, schur_launches=9.0, schur_gemm_flops=4e12, factor_ms=50.0, solve_ms=10.0,
             schur_candidate0=0.0, schur_candidate1=3.0 * (used == 'mixed'), schur_candidate2=6.0 * (used == 'mixed'))
    st0 = dict(n_active=100.0, nnz_lu=1e6, factor_flops_per_point=5e11, element_kernel_ms=1.0, scatter_kernel_ms=1.0)
    roof = bench.rooflines(_FakeEngine(), c, s, st0, used, [100.0], 4, dict(hbm_gbs=6500.0, bf16_tflops=1600.0),
                           'measured', {'fp64_dmma': 34.0, 'fp64_dmma_3m': 40.0})
    # 4 points x half of 0.5 TFLOP in 50 ms
    assert roof[0]['achieved'] == pytest.approx(20.0) and roof[0]['flops_per_sweep'] == pytest.approx(1e12)
    assert roof[0]['frac'] == pytest.approx(20.0 / (40.0 if used == 'fp64' else 800.0))
    assert roof[0]['traffic'] == (pytest.approx(4 * 5.60e9) if used == 'fp64' else None)
    text = roof[0]['kernel']
    assert 'sym_pivot_kernel' in text and 'sym_panel_kernel' in text and 'dmma' not in text and 'level' not in text
    if used == 'fp64':
        assert 'sym_schur_kernel' in text and 'tma_gemm' not in text
    else:
        assert '<64,3,true>' in text and 'for 3 updates' in text and '<128,2,true>' not in text
        assert 'SIMT FP32 64x64) for 6 updates' in text
    assert 'sym_fwd_kernel' in roof[1]['kernel']


@pytest.mark.gpu
@pytest.mark.parametrize('symmetric', [0, 1])
def test_statistics_name_the_path_that_ran(built_lib, symmetric, monkeypatch):
    monkeypatch.setenv('SS_SYMMETRIC', str(symmetric))
    c = cases.make_case('me1_64x256', seed=5, cols=16, rows=41, points=2)
    w = 2 * np.pi * c.freqs
    e = cases.engine_for(c)
    try:
        for precision in ('fp64', 'mixed'):
            _, st, _ = e.charges(w, 1.0, precision)
            s = e.stats()
            assert (st == 0).all() and s['symmetric'] == symmetric
            picks = [s[f'schur_candidate{i}'] for i in range(4)]
            if not symmetric:
                assert 0 < sum(picks) <= s['levels']
                continue
            # two points run in two groups: an update of each in one launch of the group
            assert sum(picks) == (0.0 if precision == 'fp64' else s['schur_launches'] / 2) and picks[3] == 0.0
            assert s['launches'] > s['schur_launches']
            assert s['panel_gemm_dmma'] == s['panel_thin_tiles'] == s['small_fronts'] == s['panel_tune_simt_ms'] == 0.0
    finally:
        e.close()
