"""Far wings by cells (runs of lines whose region-I wings are summed as one
series) against the oracle: both precisions, both conventions, one and several
conditions per warp, cell counts with a remainder, uneven line densities (tight
clusters, lone lines, gaps wider than the cut), pressures from Doppler- to
Lorentz-dominated, coarse and fine grids, chunks that start inside the grid.

Tolerances: FP64 1e-10 (the parity bar; the series leaves off less than 1e-15
of a line's value), mixed 1e-4 above 1e-6 of the peak and 1e-6 integrated (the
stated bound is 6.1e-5; the series' own share 1e-8).
"""
import numpy as np
import pytest

import oracle
from gpu_cross_b200 import capi, synth

from helpers import assert_fp64_parity, assert_mixed_parity, run_engine

pytestmark = pytest.mark.gpu

CUT = 25.0


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


def uneven(n, seed):
    """n lines over 1000-1100: two thirds uniform, a tight cluster, a pile of
    coinciding centres, and lone lines beyond a gap wider than the cut."""
    lines = synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    nu = lines.nu.copy()
    k = n // 6
    nu[:k] = 1050.0 + 0.3 * rng.random(k)
    nu[k:k + n // 12] = 1033.125
    nu[-7:] = np.linspace(1140.0, 1150.0, 7)
    nu[-10:-7] = [930.0, 931.0, 960.0]
    order = np.argsort(nu, kind="stable")
    lines.nu[:] = nu
    out = synth.LineList(*(np.ascontiguousarray(getattr(lines, f)[order]) if f != "nu" else np.sort(nu)
                           for f in ("nu", "energies", "aif", "gns", "gamma", "n")))
    out.gamma[::97] = 0.0  # lines without Lorentz width: region I adds nothing
    out.aif[::89] = 0.0
    return out


def reference(convention, fr, lines, cond, df, p):
    scaled = synth.LineList(lines.nu, lines.energies, lines.aif, lines.gns, lines.gamma * p, lines.n)
    f = oracle.gpu_convention if convention == capi.CONV_GPU else oracle.cpu_convention
    return f(oracle.VOIGT, fr, np.zeros_like(fr), scaled, cond, df)


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("n, df, make", [(4096, 0.01, "even"), (16385, 0.05, "even"), (30001, 0.11, "uneven"),
                                         (9001, 0.02, "uneven")])
def test_cells_one_condition(engine, cuda, convention, n, df, make):
    lines = uneven(n, 31) if make == "uneven" else synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=30)
    grid = synth.Grid(985.0, 1117.0, int(132.0 / df))
    fr = grid.freq()
    for t, p in ((296.0, 1e-3), (1500.0, 1.0), (500.0, 10.0)):
        cond = dict(temperature=t, partition=synth.partition_poly(t), mean_mass=17.03, pressure=1.0,
                    ref_temp=296.0, cut=CUT)
        ref = reference(convention, fr, lines, cond, grid.dfreq, p)
        run = dict(conds=[dict(cond, gamma_scale=p)], convention=convention)
        f64 = run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, **run)[0]
        assert_fp64_parity(f64, ref)
        mix = run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, precision=capi.MIXED, **run)[0]
        assert_mixed_parity(mix, ref)
        # every launch shape and split count sums the same cells
        for kw in (dict(P=1, W=8), dict(P=8, S=3), dict(P=2, S=7)):
            assert_fp64_parity(run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, **run, **kw)[0], ref)
            assert_mixed_parity(run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda,
                                           precision=capi.MIXED, **run, **kw)[0], ref)


@pytest.mark.parametrize("C", [2, 4, 8])
@pytest.mark.parametrize("n, df", [(8003, 0.1), (6000, 0.021), (40001, 0.1)])
def test_cells_groups_of_conditions(engine, cuda, C, n, df):
    lines = uneven(n, 33)
    grid = synth.Grid(985.0, 1117.0, int(132.0 / df))
    fr = grid.freq()
    base = dict(mean_mass=17.03, pressure=1.0, ref_temp=296.0, cut=CUT)
    conds = [dict(base, temperature=t, partition=synth.partition_poly(t), gamma_scale=p)
             for t in (300.0, 2100.0) for p in (1e-3, 0.1, 1.0, 10.0)]
    refs = [reference(capi.CONV_GPU, fr, lines, c, grid.dfreq, c["gamma_scale"]) for c in conds]
    for kw in (dict(), dict(S=5), dict(W=8) if C < 8 else dict(S=2)):
        f64 = run_engine(engine, capi.VOIGT, lines, fr, base, grid.dfreq, cuda, conds=conds, C=C, **kw)
        mix = run_engine(engine, capi.VOIGT, lines, fr, base, grid.dfreq, cuda, conds=conds, C=C,
                         precision=capi.MIXED, **kw)
        for k in range(len(conds)):
            assert_fp64_parity(f64[k], refs[k])
            assert_mixed_parity(mix[k], refs[k])


def test_cells_chunk_inside_the_grid(engine, cuda):
    lines = uneven(12000, 35)
    grid = synth.Grid(985.0, 1117.0, 6601)
    fr = grid.freq()
    cond = dict(temperature=900.0, partition=synth.partition_poly(900.0), mean_mass=17.03, pressure=1.0,
                ref_temp=296.0, cut=CUT)
    ref = reference(capi.CONV_GPU, fr, lines, cond, grid.dfreq, 1.0)
    for start, points in ((0, 1), (1234, 3333), (6600, 1)):
        got = run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, conds=[dict(cond, gamma_scale=1.0)],
                         start_idx=start, points=points)[0]
        assert_fp64_parity(got[start:start + points], ref[start:start + points])
        assert not got[:start].any() and not got[start + points:].any()


@pytest.mark.parametrize("C", [1, 4])
def test_cells_low_wavenumbers(engine, cuda, C):
    """Lines from 0 to 60 cm-1: Doppler widths of a few 1e-5
    cm-1 and less, so the cut reaches x ~ 1e6 and beyond: wide lines, and cells
    that no series may stand for."""
    lines = synth.random_lines(9001, 0.001, 60.0, 2500.0, 1e-6, 1e2, seed=41)
    grid = synth.Grid(0.5, 70.5, 7000)
    fr = grid.freq()
    base = dict(mean_mass=17.03, pressure=1.0, ref_temp=296.0, cut=CUT)
    conds = [dict(base, temperature=t, partition=synth.partition_poly(t), gamma_scale=p)
             for t in (300.0, 2100.0) for p in (1e-2, 1.0)]
    f64 = run_engine(engine, capi.VOIGT, lines, fr, base, grid.dfreq, cuda, conds=conds, C=C)
    mix = run_engine(engine, capi.VOIGT, lines, fr, base, grid.dfreq, cuda, conds=conds, C=C, precision=capi.MIXED)
    for k, c in enumerate(conds):
        ref = reference(capi.CONV_GPU, fr, lines, c, grid.dfreq, c["gamma_scale"])
        assert_fp64_parity(f64[k], ref)
        assert_mixed_parity(mix[k], ref)


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("n, df, make", [(60001, 0.1, "even"), (60001, 0.1, "uneven"), (16385, 0.04, "uneven")])
def test_cells_single_condition_tiles(engine, cuda, convention, n, df, make):
    """Single conditions at the default shape on 8-point tiles (a coarse grid over a dense list: a 32-point row
    holds more lines than four cells) and on 16-point ones, both above the 1.2e7 pairs from which cells are used."""
    lines = uneven(n, 51) if make == "uneven" else synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=50)
    grid = synth.Grid(985.0, 1117.0, int(132.0 / df))
    fr = grid.freq()
    for t, p in ((296.0, 1e-3), (1500.0, 10.0)):
        cond = dict(temperature=t, partition=synth.partition_poly(t), mean_mass=17.03, pressure=1.0,
                    ref_temp=296.0, cut=CUT)
        ref = reference(convention, fr, lines, cond, grid.dfreq, p)
        run = dict(conds=[dict(cond, gamma_scale=p)], convention=convention)
        assert_fp64_parity(run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, **run)[0], ref)
        assert_mixed_parity(run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda,
                                       precision=capi.MIXED, **run)[0], ref)
