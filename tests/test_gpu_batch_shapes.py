"""Batches of which the caller names the points per thread but not the conditions per
warp."""
import pytest
import torch

from gpu_cross_b200 import capi, synth

from helpers import assert_mixed_parity, run_engine, to_device

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("P", [2, 4, 8])
def test_wide_tiles_asked_for_keep_the_group_kernel(engine, cuda, P):
    """A mixed batch runs in groups of two conditions then (the group kernel takes no
    tile width): grid check, step one, moments, step two and core pass make five
    launches.  One condition at a time on wide tiles would go line by line."""
    lines = synth.random_lines(40000, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=97)
    grid = synth.Grid(985.0, 1117.0, 13200)
    base = dict(partition=synth.partition_poly(700.0), temperature=700.0, mean_mass=17.03, pressure=1.0,
                ref_temp=296.0, cut=25.0)
    conds = [dict(base, gamma_scale=p) for p in (0.1, 1.0)]
    dev = to_device(lines, cuda)
    dfr = torch.as_tensor(grid.freq(), device=cuda)
    out = torch.zeros((2, grid.npoints), dtype=torch.float64, device=cuda)
    opts = capi.make_options(capi.VOIGT, grid.dfreq, 17.03, precision=capi.MIXED, points_per_thread=P, line_splits=1)
    cc = [capi.make_condition(700.0, base["partition"], 1.0, c["gamma_scale"], 25.0) for c in conds]
    engine.set_stream(torch.cuda.current_stream(cuda).cuda_stream)
    g = engine.capture(opts, cc, capi.make_lines(dev), capi.make_grid(dfr), out.data_ptr(), grid.npoints)
    try:
        assert g.kernel_count() == 5
        g.launch(torch.cuda.current_stream(cuda).cuda_stream)
        torch.cuda.synchronize(cuda)
    finally:
        g.close()
    ref = run_engine(engine, capi.VOIGT, lines, grid.freq(), base, grid.dfreq, cuda, conds=conds)
    got = out.cpu().numpy()
    for k in range(2):
        assert_mixed_parity(got[k], ref[k])


@pytest.mark.parametrize("ncond, n, df", [(8, 40000, 0.01), (4, 40000, 0.05), (6, 9000, 0.02), (3, 40000, 0.01)])
def test_batches_go_in_the_largest_groups(engine, cuda, ncond, n, df):
    """Grid check, step one, moments, step two and the core pass: groups of 8, 4 and 2
    conditions; 3 go one at a time, without a core pass of their own."""
    lines = synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=99)
    grid = synth.Grid(985.0, 1117.0, int(132.0 / df))
    base = dict(mean_mass=17.03, pressure=1.0, ref_temp=296.0, cut=25.0)
    conds = [dict(base, temperature=300.0 + 200.0 * k, partition=synth.partition_poly(300.0 + 200.0 * k),
                  gamma_scale=10.0 ** (k % 4 - 2)) for k in range(ncond)]
    dev = to_device(lines, cuda)
    dfr = torch.as_tensor(grid.freq(), device=cuda)
    out = torch.zeros((ncond, grid.npoints), dtype=torch.float64, device=cuda)
    opts = capi.make_options(capi.VOIGT, grid.dfreq, 17.03, precision=capi.MIXED, line_splits=1)
    cc = [capi.make_condition(c["temperature"], c["partition"], 1.0, c["gamma_scale"], 25.0) for c in conds]
    engine.set_stream(torch.cuda.current_stream(cuda).cuda_stream)
    g = engine.capture(opts, cc, capi.make_lines(dev), capi.make_grid(dfr), out.data_ptr(), grid.npoints)
    try:
        assert g.kernel_count() == (4 if ncond == 3 else 5)
        g.launch(torch.cuda.current_stream(cuda).cuda_stream)
        torch.cuda.synchronize(cuda)
    finally:
        g.close()
    ref = run_engine(engine, capi.VOIGT, lines, grid.freq(), base, grid.dfreq, cuda, conds=conds)
    got = out.cpu().numpy()
    for k in range(ncond):
        assert_mixed_parity(got[k], ref[k])
