"""Mixed precision where whole cells of lines are far weaker than the rest: the
strongest intensity of a stretch between 1e-36 and 1e-45 (a cold condition on a
hot list), lines of intensity 0 and lines without Lorentz width among them.  The
result has to be finite everywhere and within the mixed bound of the FP64 one
(1e-4 above 1e-6 of the peak, 1e-6 integrated; the stated bound is 6.1e-5)."""
import math

import numpy as np
import pytest
import torch

from gpu_cross_b200 import capi, synth

from helpers import assert_mixed_parity, run_engine

pytestmark = pytest.mark.gpu

T, MASS, CUT = 300.0, 17.03, 25.0
GRID = synth.Grid(985.0, 1117.0, 6600)


@pytest.fixture(scope="module")
def engine(cuda):
    e = capi.Engine(0)
    yield e
    e.close()


def aif_for(s, nu):
    """A that gives intensity s at E'' = 0, g = 1 (Voigt, GPU convention)."""
    cmcoef = 1.0 / (8.0 * math.pi * 2.99792458e10)
    beta = 6.6260693e-27 * 2.99792458e10 / (1.380658e-16 * T)
    return s * nu * nu * synth.partition_poly(T) / (cmcoef * 0.564189584 * (1.0 - np.exp(-beta * nu)))


def with_weak_stretch(s, n=40000, seed=61, everywhere=False):
    lines = synth.random_lines(n, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=seed)
    weak = np.ones(n, bool) if everywhere else (lines.nu > 1040.0) & (lines.nu < 1065.0)
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    lines.energies[weak] = 0.0
    lines.gns[weak] = 1
    lines.aif[weak] = aif_for(s, lines.nu[weak]) * 10.0 ** rng.uniform(-3.0, 0.0, weak.sum())
    at = np.flatnonzero(weak)
    lines.aif[at[::7]] = 0.0
    lines.gamma[at[::5]] = 0.0
    return lines


def conditions(count):
    base = dict(temperature=T, partition=synth.partition_poly(T), mean_mass=MASS, pressure=1.0, ref_temp=296.0,
                cut=CUT)
    return [dict(base, gamma_scale=p) for p in (1.0, 1e-3, 0.1, 10.0, 0.01, 0.3, 3.0, 0.03)[:count]]


@pytest.mark.parametrize("C", [1, 2, 4, 8])
@pytest.mark.parametrize("s", [1e-36, 5e-39, 1e-39, 1e-42, 1e-45])
def test_weak_stretch_beside_strong_lines(engine, cuda, s, C):
    lines, conds = with_weak_stretch(s), conditions(C)
    run = dict(conds=conds, C=C)
    ref = run_engine(engine, capi.VOIGT, lines, GRID.freq(), conds[0], GRID.dfreq, cuda, **dict(run, C=0))
    got = run_engine(engine, capi.VOIGT, lines, GRID.freq(), conds[0], GRID.dfreq, cuda, precision=capi.MIXED, **run)
    assert np.isfinite(got).all()
    for k in range(C):
        assert_mixed_parity(got[k], ref[k])


@pytest.mark.parametrize("s", [1e-36, 1e-39, 1e-42, 1e-45])
def test_only_weak_lines(engine, cuda, s):
    """Nothing but weak lines: finite, and no larger than the FP64 result by more
    than what FP32 holds below its normal range (2^-150 per line and point)."""
    lines, cond = with_weak_stretch(s, everywhere=True), conditions(1)[0]
    ref = run_engine(engine, capi.VOIGT, lines, GRID.freq(), cond, GRID.dfreq, cuda, conds=[cond])[0]
    got = run_engine(engine, capi.VOIGT, lines, GRID.freq(), cond, GRID.dfreq, cuda, conds=[cond],
                     precision=capi.MIXED)[0]
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) <= 1e-4 * ref + 40000 * 2.0 ** -149).all()


@pytest.mark.parametrize("s", [1e-36, 1e-39, 1e-42])
def test_weak_stretch_streamed(engine, cuda, s):
    lines = with_weak_stretch(s)
    s32 = (lines.aif * lines.gns * np.exp(-1.4387752 * lines.energies / T) / aif_for(1.0, lines.nu)).astype(np.float32)
    host = [torch.from_numpy(x).pin_memory() for x in (lines.nu, s32, lines.gamma.astype(np.float32))]
    fr = torch.as_tensor(GRID.freq(), device=cuda)
    res = []
    for prec in (capi.FP64, capi.MIXED):
        out = torch.zeros(GRID.npoints, dtype=torch.float64, device=cuda)
        engine.set_stream(torch.cuda.current_stream(cuda).cuda_stream)
        engine.stream_execute(capi.make_options(capi.VOIGT, GRID.dfreq, MASS, precision=prec),
                              capi.make_condition(T, synth.partition_poly(T), 1.0, 1.0, CUT), host[0].data_ptr(),
                              host[1].data_ptr(), host[2].data_ptr(), lines.nu.size, capi.make_grid(fr),
                              out.data_ptr(), 1 << 20)
        res.append(out.cpu().numpy())
    assert np.isfinite(res[1]).all()
    assert_mixed_parity(res[1], res[0])


@pytest.mark.parametrize("s", [1e-39, 1e-42])
def test_weak_stretch_served(cuda, s):
    lines = with_weak_stretch(s)
    srv = capi.Server(0, lanes=2)
    try:
        mid = srv.add_molecule(lines, MASS)
        res = []
        for prec in (capi.FP64, capi.MIXED):
            rid = srv.submit(mid, capi.VOIGT, prec, T, synth.partition_poly(T), 1.0, 985.0, GRID.dfreq, GRID.npoints,
                             cut=CUT)
            res.append(srv.wait(rid, GRID.npoints)[0])
    finally:
        srv.close()
    assert np.isfinite(res[1]).all()
    assert_mixed_parity(res[1], res[0])
