"""Single conditions whose far wings go by cells (runs of lines summed as one
series), with the lines of a tile split over 2 to 64 parts -- more parts than a
window has cells among them -- and with 4 and 8 warps per block, on 16- and 8-point
tiles.  Every case asserts that cells are used: step one, moments, step two and the
split sums make five launches with the grid check.

Tolerances: FP64 1e-12, the stated bound (summation order, reciprocals, the series'
rest of 3e-15 of a line); mixed 1e-4 above 1e-6 of the peak and 1e-6 integrated
(the stated bound is 6.1e-5)."""
import numpy as np
import pytest
import torch

import oracle
from gpu_cross_b200 import capi, synth

from helpers import assert_fp64_parity, assert_mixed_parity, to_device

pytestmark = pytest.mark.gpu

CUT = 25.0
# lines, grid step: 4500 lines per window on 16-point tiles, 16000 on 8-point ones
SIZES = [(16385, 0.02), (60001, 0.1)]


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


_made = {}


def case(n, df):
    if (n, df) not in _made:
        lines = synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=95)
        grid = synth.Grid(985.0, 1117.0, int(132.0 / df))
        cond = dict(temperature=700.0, partition=synth.partition_poly(700.0), mean_mass=17.03, pressure=1.0,
                    ref_temp=296.0, cut=CUT)
        fr = grid.freq()
        _made[n, df] = lines, grid, fr, cond, oracle.gpu_convention(oracle.VOIGT, fr, np.zeros_like(fr), lines, cond,
                                                                    grid.dfreq)
    return _made[n, df]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("n, df", SIZES)
@pytest.mark.parametrize("S, W", [(2, 4), (3, 8), (7, 4), (64, 4), (64, 8)])
def test_cells_in_parts(engine, cuda, precision, n, df, S, W):
    lines, grid, fr, cond, ref = case(n, df)
    dev = to_device(lines, cuda)
    dfr = torch.as_tensor(fr, device=cuda)
    out = torch.zeros(len(fr), dtype=torch.float64, device=cuda)
    opts = capi.make_options(capi.VOIGT, grid.dfreq, cond["mean_mass"], precision=precision, points_per_thread=1,
                             warps_per_block=W, conditions_per_warp=1, line_splits=S)
    cc = [capi.make_condition(cond["temperature"], cond["partition"], 1.0, 1.0, CUT)]
    engine.set_stream(torch.cuda.current_stream(cuda).cuda_stream)
    g = engine.capture(opts, cc, capi.make_lines(dev), capi.make_grid(dfr), out.data_ptr(), len(fr))
    try:
        assert g.kernel_count() == 5
        g.launch(torch.cuda.current_stream(cuda).cuda_stream)
        engine.sync()
        torch.cuda.synchronize(cuda)
    finally:
        g.close()
    got = out.cpu().numpy()
    if precision == capi.FP64:
        assert_fp64_parity(got, ref, rel=1e-12)
    else:
        assert_mixed_parity(got, ref)


@pytest.mark.parametrize("n, df", SIZES)
def test_cells_in_the_cpu_convention_and_from_a_split_count_of_one(engine, cuda, n, df):
    lines, grid, fr, cond, _ = case(n, df)
    ref = oracle.cpu_convention(oracle.VOIGT, fr, np.zeros_like(fr), lines, cond, grid.dfreq)
    dev = to_device(lines, cuda)
    dfr = torch.as_tensor(fr, device=cuda)
    engine.set_stream(torch.cuda.current_stream(cuda).cuda_stream)
    for S, kernels in ((1, 4), (5, 5)):
        out = torch.zeros(len(fr), dtype=torch.float64, device=cuda)
        opts = capi.make_options(capi.VOIGT, grid.dfreq, cond["mean_mass"], convention=capi.CONV_CPU, line_splits=S)
        cc = [capi.make_condition(cond["temperature"], cond["partition"], 1.0, 1.0, CUT)]
        g = engine.capture(opts, cc, capi.make_lines(dev), capi.make_grid(dfr), out.data_ptr(), len(fr))
        try:
            assert g.kernel_count() == kernels
            g.launch(torch.cuda.current_stream(cuda).cuda_stream)
            torch.cuda.synchronize(cuda)
        finally:
            g.close()
        assert_fp64_parity(out.cpu().numpy(), ref, rel=1e-12)
