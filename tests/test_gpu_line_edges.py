"""Voigt lines at the edges of what a list or a condition may hold, single
conditions and batches, on calls below and above the pair count from which far
wings go by cells."""
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


def conditions(count, **kw):
    base = dict(temperature=300.0, partition=synth.partition_poly(300.0), mean_mass=17.03, pressure=1.0, ref_temp=296.0,
                cut=25.0)
    return [dict(base, gamma_scale=p, **kw) for p in (0.1, 1.0)[:count]]


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("n, points", [(300, 4001), (20000, 7000)])
@pytest.mark.parametrize("C", [1, 2])
def test_line_at_zero_wavenumber(engine, cuda, convention, n, points, C):
    """A centre of 0 in reach of the grid.  GPU convention: its Doppler width is
    0, x infinite, and a mixed call leaves it out (FP64 gives the reference's NaN
    there), so the FP64 spectrum of the other lines is the reference; the CPU
    convention takes the centre as 1e-6."""
    lines = synth.random_lines(n, 1.0, 60.0, 2500.0, 1e-6, 1e2, seed=71)
    lines.nu[0] = 0.0
    grid = synth.Grid(0.5, 0.5 + points * 0.01, points)
    conds = conditions(C)
    args = (grid.freq(), conds[0], grid.dfreq, cuda)
    run = dict(conds=conds, C=C, convention=convention)
    rest = lines.slice(1, n) if convention == capi.CONV_GPU else lines
    ref = run_engine(engine, capi.VOIGT, rest, *args, **dict(run, C=0))
    got = run_engine(engine, capi.VOIGT, lines, *args, precision=capi.MIXED, **run)
    assert np.isfinite(got).all()
    for k in range(C):
        assert_mixed_parity(got[k], ref[k])


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("C, P", [(1, 0), (1, 1), (1, 2), (2, 0)])
def test_negative_cut_reaches_nothing(engine, cuda, convention, precision, C, P):
    """The cut rule gives 25 P: a negative pressure leaves every window empty."""
    lines = synth.random_lines(400, 1000.0, 1040.0, 2500.0, 1e-6, 1e2, seed=73)
    grid = synth.Grid(995.0, 1045.0, 5000)
    for pressure in (-1e-4, -0.02, -1.0):
        conds = conditions(C, cut=-1.0)
        for c in conds:
            c["pressure"] = pressure
        got = run_engine(engine, capi.VOIGT, lines, grid.freq(), conds[0], grid.dfreq, cuda, conds=conds, C=C, P=P,
                         convention=convention, precision=precision)
        assert not got.any()


@pytest.mark.parametrize("temperatures", [1, 7, 8, 9, 16])
def test_batches_of_distinct_temperatures(engine, cuda, temperatures):
    """Step one keeps the values of up to 16 temperatures per line in shared
    memory, 6 KB each beside its own 4 KB: 8 of them cross 48 KB."""
    lines = synth.random_lines(3000, 1000.0, 1040.0, 2500.0, 1e-6, 1e2, seed=75)
    grid = synth.Grid(995.0, 1045.0, 500)
    conds = [dict(c, temperature=t, partition=synth.partition_poly(t))
             for t in np.linspace(250.0, 2500.0, temperatures) for c in conditions(2)]
    args = (grid.freq(), conds[0], grid.dfreq, cuda)
    ref = run_engine(engine, capi.VOIGT, lines, *args, conds=conds)
    got = run_engine(engine, capi.VOIGT, lines, *args, conds=conds, C=2, precision=capi.MIXED)
    for k in range(len(conds)):
        assert_mixed_parity(got[k], ref[k])


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("C, P", [(1, 0), (1, 1), (1, 2), (1, 4), (1, 8), (2, 0)])
def test_strong_lines_far_beyond_their_doppler_width(engine, cuda, convention, C, P):
    """Strong lines at 1e-6 cm-1, where the Doppler width is some 1e-12: x reaches 1e13
    inside the window, u = x^2 + y^2 - 1/2 is 1e26 and u times the amplitude beyond the
    FP32 range."""
    lines = synth.random_lines(500, 1.0, 60.0, 2500.0, 1e-6, 1e2, seed=77)
    lines.nu[:9] = np.linspace(1e-6, 2e-6, 9)
    lines.aif[:9] = 1e8
    lines.gns[:9] = 100
    grid = synth.Grid(18.0, 58.0, 4000)
    conds = [dict(c, cut=100.0) for c in conditions(2)]
    args = (grid.freq(), conds[0], grid.dfreq, cuda)
    run = dict(conds=conds, convention=convention)
    ref = run_engine(engine, capi.VOIGT, lines, *args, **run)
    got = run_engine(engine, capi.VOIGT, lines, *args, C=C, P=P, precision=capi.MIXED, **run)
    assert np.isfinite(got).all()
    for k in range(2):
        assert_mixed_parity(got[k], ref[k])
