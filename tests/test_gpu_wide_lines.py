"""Mixed precision on lines whose window spans more than 5e4 Doppler widths (low
wavenumbers, a cut of 100): a reciprocal per pair, in every layout, calls with and
without cells, beside lines beyond 1e8 widths and beside ordinary ones, at pressures
from Doppler- to Lorentz-dominated.  Against FP64 in the mixed bound (1e-4 above 1e-6
of the peak, 1e-6 integrated)."""
import numpy as np
import pytest

from gpu_cross_b200 import capi, synth

from helpers import assert_mixed_parity, run_engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("C, P", [(1, 1), (1, 2), (2, 0), (4, 0), (8, 0)])
@pytest.mark.parametrize("n, f0, points, df", [(150, 2.0, 9000, 0.01), (3000, 200.0, 12001, 0.01), (30000, 5.0, 1500, 0.1),
                                               (700, 0.01, 3000, 0.003)])
def test_windows_of_many_doppler_widths(engine, cuda, C, P, n, f0, points, df):
    span = points * df
    lines = synth.random_lines(n, f0, f0 + span, 2500.0, 1e-6, 1e2, seed=87)
    lines.nu[:5] = f0 * np.linspace(1e-6, 1.0, 5)  # x beyond 1e8 at the first
    lines.gamma[::11] = 0.0
    grid = synth.Grid(f0 + 0.1 * span, f0 + 1.1 * span, points)
    base = dict(mean_mass=17.03, pressure=1.0, ref_temp=296.0, cut=100.0)
    conds = [dict(base, temperature=t, partition=synth.partition_poly(t), gamma_scale=p)
             for t in (300.0, 2100.0) for p in (1e-4, 0.1, 1.0, 40.0)]
    run = dict(conds=conds)
    args = (grid.freq(), conds[0], grid.dfreq, cuda)
    ref = run_engine(engine, capi.VOIGT, lines, *args, **run)
    got = run_engine(engine, capi.VOIGT, lines, *args, C=C, P=P, precision=capi.MIXED, **run)
    assert np.isfinite(got).all()
    for k in range(len(conds)):
        assert_mixed_parity(got[k], ref[k])
