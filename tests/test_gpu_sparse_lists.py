"""FP64 Voigt on lists so sparse that a 32-point row has from no line to a few whose
core reaches it (taken a lane per point) and, around clusters, many (a lane per line),
on every tile width and split count, against the oracle (1e-10, the parity bar)."""
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


def sparse(n, seed):
    """n lines over 1000-1060, then clusters of 1 to 6 lines within 0.02 cm-1."""
    lines = synth.random_lines(n + 21, 1000.0, 1060.0, 2500.0, 1e-6, 1e2, seed=seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    at = 1005.0 + 9.0 * np.arange(6)
    clustered = np.concatenate([at[k] + 0.02 * rng.random(k + 1) for k in range(6)])
    nu = np.concatenate([1000.0 + 60.0 * rng.random(n), clustered])
    order = np.argsort(nu, kind="stable")
    for f in ("energies", "aif", "gns", "gamma", "n"):
        getattr(lines, f)[:] = getattr(lines, f)[order]
    lines.nu[:] = nu[order]
    return lines


@pytest.mark.parametrize("convention", [capi.CONV_GPU, capi.CONV_CPU])
@pytest.mark.parametrize("n, df", [(3, 0.005), (60, 0.002), (400, 0.01), (1500, 0.05)])
def test_few_cores_per_row(engine, cuda, convention, n, df):
    lines = sparse(n, 83)
    grid = synth.Grid(998.0, 1062.0, int(64.0 / df))
    fr = grid.freq()
    f = oracle.gpu_convention if convention == capi.CONV_GPU else oracle.cpu_convention
    for t, p in ((296.0, 1e-3), (1500.0, 1.0)):
        cond = dict(temperature=t, partition=synth.partition_poly(t), mean_mass=17.03, pressure=1.0, ref_temp=296.0,
                    cut=25.0)
        scaled = synth.LineList(lines.nu, lines.energies, lines.aif, lines.gns, lines.gamma * p, lines.n)
        ref = f(oracle.VOIGT, fr, np.zeros_like(fr), scaled, cond, grid.dfreq)
        for P, S in ((0, 0), (2, 1), (4, 1), (8, 3), (2, 5), (1, 1)):
            got = run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, convention=convention, P=P, S=S,
                             conds=[dict(cond, gamma_scale=p)])[0]
            assert_fp64_parity(got, ref)
        got = run_engine(engine, capi.VOIGT, lines, fr, cond, grid.dfreq, cuda, convention=convention, C=2,
                         conds=[dict(cond, gamma_scale=p)] * 2)
        assert_fp64_parity(got[0], ref)
        assert_fp64_parity(got[1], ref)
