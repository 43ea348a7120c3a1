"""Calls whose far-wing cells do not fit the engine's scratch (a limit set on the
engine stands for a full card): the same spectrum line by line, no reallocation on
repeated calls, and captured as they run."""
import pytest
import torch

from gpu_cross_b200 import capi, synth

from helpers import assert_fp64_parity, assert_mixed_parity, to_device

pytestmark = pytest.mark.gpu

N, MASS, DF = 40001, 17.03, 0.02


class Call:
    """One call on resident buffers: 11000 lines per window, 7e7 pairs and more."""

    def __init__(self, device, precision, ncond, C):
        lines = synth.random_lines(N, 1000.0, 1100.0, 2500.0, 1e-6, 1e2, seed=81)
        self.grid = synth.Grid(985.0, 1117.0, int(132.0 / DF))
        self.dev = to_device(lines, device)
        self.fr = torch.as_tensor(self.grid.freq(), device=device)
        self.out = torch.zeros((ncond, self.grid.npoints), dtype=torch.float64, device=device)
        opts = capi.make_options(capi.VOIGT, self.grid.dfreq, MASS, precision=precision, conditions_per_warp=C)
        conds = [capi.make_condition(t, synth.partition_poly(t), 1.0, 1.0, 25.0) for t in (300.0, 1500.0)[:ncond]]
        self.args = (opts, conds, capi.make_lines(self.dev), capi.make_grid(self.fr), self.out.data_ptr(),
                     self.grid.npoints)

    def run(self, engine):
        self.out.zero_()
        engine.set_stream(torch.cuda.current_stream(self.out.device).cuda_stream)
        engine.execute(*self.args)
        engine.sync()
        return self.out.cpu().numpy()

    def replay(self, engine):
        g = engine.capture(*self.args)
        try:
            self.out.zero_()
            g.launch(torch.cuda.current_stream(self.out.device).cuda_stream)
            torch.cuda.synchronize(self.out.device)
            return self.out.cpu().numpy(), g.kernel_count()
        finally:
            g.close()


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("ncond, C", [(1, 1), (2, 2)])
def test_cells_without_room(cuda, precision, ncond, C):
    call = Call(cuda, precision, ncond, C)
    free = capi.Engine(0)
    tight = capi.Engine(0)
    try:
        want, kernels = call.replay(free)
        need = free.scratch_bytes()
        tight.limit_scratch(need - 1)
        got, k = call.replay(tight)  # captured first
        held = tight.scratch_bytes()
        assert 0 < held < need
        assert k == kernels - 1  # no moments
        check = assert_fp64_parity if precision == capi.FP64 else assert_mixed_parity
        for c in range(ncond):
            check(got[c], want[c])
        for _ in range(2):
            assert (call.run(tight) == got).all()
            assert tight.scratch_bytes() == held
        assert (call.replay(tight)[0] == got).all()
        # room again: the cells come back
        tight.limit_scratch(0)
        assert (call.run(tight) == want).all()
        assert tight.scratch_bytes() == need
    finally:
        free.close()
        tight.close()


def test_records_without_room(cuda):
    call = Call(cuda, capi.MIXED, 1, 1)
    e = capi.Engine(0)
    try:
        e.limit_scratch(1 << 20)
        with pytest.raises(capi.XsError) as info:
            call.run(e)
        assert info.value.code == capi.XS_ERR_NOMEM
        e.limit_scratch(0)
        assert call.run(e).any()
    finally:
        e.close()
