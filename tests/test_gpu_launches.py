"""The launch counts that runs report, against the kernels that the profiler
records: every kernel of the work is counted, and no other (the pointer and
counter set-up of a run is not).  Marked ``gpu``; run on a B200."""
import numpy as np
import pytest

from temf3dt_b200 import fetd
from tests.golden_cases import adjoint_misfit_case, cell_grid_2x2x2, small_synth, synth_oracle_model, tiny_synth

pytestmark = pytest.mark.gpu


def _recorded(work):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        out = work()
    names = [e.name for e in p.events() if "temf::k_" in e.name]
    if not names:
        pytest.skip("the profiler records no kernels here")
    return out, sum(1 for n in names if "k_set_ptr" not in n and "k_set_int" not in n)


def _args(m):
    return m.ctl.sp_division, m.ctl.sp_double, m.ctl.sp_dblesize, m.ctl.time_maximum


def test_run_and_adjoint_count_their_kernels():
    m = small_synth()
    g = fetd.FetdGPU(0)
    fetd.load_case(g, m.mesh, m.ctl)
    g.run(*_args(m))  # the first run picks the sweeps' schedule, which is not counted
    out, n = _recorded(lambda: g.run(*_args(m)))
    assert len(out.trial_accepted) > 0 and out.n_launch == n
    g.adjoint_record(5)
    out = g.run(*_args(m))
    d_obs, mask = adjoint_misfit_case(out.fields)
    cell = cell_grid_2x2x2(synth_oracle_model(m))
    (_, _, tm), n = _recorded(lambda: g.adjoint(mask * (out.fields - d_obs), cell, 8))
    assert tm["launches"] == n
    g.close()


def test_batch_counts_its_kernels():
    models = []
    for m in (tiny_synth(), small_synth()):
        g = fetd.FetdGPU(0)
        fetd.load_case(g, m.mesh, m.ctl)
        models.append(g)
    with fetd.FetdBatch(models) as b:
        args = (10, 12, 2, 1e-2)
        b.run(*args, max_steps=20)
        _, n = _recorded(lambda: b.run(*args, max_steps=20))
        assert b.timing()["launches"] == n
    for g in models:
        g.close()
