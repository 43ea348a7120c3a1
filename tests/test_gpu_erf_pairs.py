"""Doppler and Gaussian step two, whose lanes take numbered (line, point) pairs:
against the oracle where the numbering can go wrong -- lines without a point in
the tile, lines wider than a tile, piles of coinciding centres, a last tile of one
point, chunks inside the grid, more parts than lines.

Tolerance: the FP64 parity bar, 1e-10 (the same arithmetic per pair as the oracle;
only the order of the sums differs).
"""
import numpy as np
import pytest

import oracle
from gpu_cross_b200 import capi, synth

from helpers import assert_fp64_parity, run_engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


def listing(n, seed):
    """n lines over 1000-1010, a third of them on one centre, some beyond the grid."""
    lines = synth.random_lines(n, 1000.0, 1010.0, 2500.0, 1e-6, 1e2, seed=seed)
    lines.nu[n // 3:2 * n // 3] = 1004.4371
    lines.nu[-1] = 1013.0
    return lines.sorted()


@pytest.mark.parametrize("profile, convention", [(capi.DOPPLER, capi.CONV_GPU), (capi.DOPPLER, capi.CONV_CPU),
                                                 (capi.GAUSSIAN, capi.CONV_GPU)])
@pytest.mark.parametrize("n, points", [(1, 33), (2, 1), (31, 400), (33, 1025), (400, 65)])
def test_erf_pairs(engine, cuda, profile, convention, n, points):
    lines = listing(n, 61 + n)
    grid = synth.Grid(999.5, 1011.0, points)
    fr = grid.freq()
    cond = dict(temperature=700.0, partition=synth.partition_poly(700.0), mean_mass=17.03, pressure=1.0,
                ref_temp=296.0, half_width=0.01)
    oprof = {capi.DOPPLER: oracle.DOPPLER, capi.GAUSSIAN: oracle.GAUSSIAN}[profile]
    f = oracle.gpu_convention if convention == capi.CONV_GPU else oracle.cpu_convention
    ref = f(oprof, fr, np.zeros_like(fr), lines, cond, grid.dfreq)
    for kw in (dict(), dict(P=2, W=8), dict(P=1, W=8, S=5), dict(P=2, W=4, S=64)):
        got = run_engine(engine, profile, lines, fr, cond, grid.dfreq, cuda, convention=convention,
                         half_width=cond["half_width"], **kw)
        assert_fp64_parity(got, ref)
    a, m = points // 3, max(1, points // 2)
    got = run_engine(engine, profile, lines, fr, cond, grid.dfreq, cuda, convention=convention,
                     half_width=cond["half_width"], start_idx=a, points=m)
    # a chunk's windows end at its edges
    part = f(oprof, fr, np.zeros_like(fr), lines, cond, grid.dfreq, points=m, start_idx=a)
    assert_fp64_parity(got[a:a + m], part[a:a + m])
