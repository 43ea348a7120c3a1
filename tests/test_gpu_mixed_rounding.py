"""Rounding of the mixed kernels' FP32 sums, against the FP64 path in the 2-norm.

At 10 atm every line is wide and each point sums hundreds of lines of like size,
so what is left of the error is the FP32 partial sums, not one line's own
rounding."""
import numpy as np
import pytest

from gpu_cross_b200 import capi, synth

from helpers import run_engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


# Bound: the error, on the same lists, of point-parallel kernels that sum at most 32
# lines in FP32 and add those sums up with compensation.
@pytest.mark.parametrize("C, n, lo, hi, df, bound", [
    (8, 1_000_000, 500.0, 8000.0, 0.1, 5.08e-8),
    (4, 1_000_000, 500.0, 8000.0, 0.1, 5.08e-8),
    (2, 300_000, 2000.0, 2200.0, 0.01, 1.77e-8),
    (0, 300_000, 2000.0, 2200.0, 0.004, 1.77e-8),
    (0, 100_000, 1000.0, 1200.0, 0.01, 2.74e-8),
])
def test_sums_of_many_wide_lines(engine, cuda, C, n, lo, hi, df, bound):
    lines = synth.random_lines(n, lo, hi, 2500.0, 1e-6, 1e2, seed=91)
    grid = synth.Grid(lo, hi, int(round((hi - lo) / df)))
    conds = [dict(temperature=t, partition=synth.partition_poly(t), mean_mass=17.03, pressure=1.0, gamma_scale=10.0,
                  ref_temp=296.0, cut=25.0) for t in np.repeat(np.linspace(300.0, 2400.0, 4), 2)]
    args = (grid.freq(), conds[0], grid.dfreq, cuda)
    ref = run_engine(engine, capi.VOIGT, lines, *args, conds=conds)
    got = run_engine(engine, capi.VOIGT, lines, *args, conds=conds, C=C, precision=capi.MIXED)
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    rms = float(np.sqrt(np.mean(err * err)))
    assert rms <= bound, f"rms error {rms:.3e}"
