"""The autotuner's search over the BLKTRI-order path's stage schedules: its four
alternatives are timed where they differ, for plans that divide; for plans with a
pivot table they are one launch, and the schedule stays as it is."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table,candidates", [(-1, 1), (0, 5)])
def test_candidates(chylib, table, candidates):
    plan = chylib.Plan(chylib.grid(66, 16, 32), "blktri", 1, pivot_table_max=table)
    rho = chylib.to_cuda_fortran(synth.disk_density(66, 16, 32, 5, spiral=True, spectrum=True))
    t = chylib.autotune_multi([plan], [rho], repeats=1)
    assert t["candidates"] == candidates
    if table:
        assert (t["blk_warps"], t["blk_ctas_per_sm"]) == (8, 2) and plan.schedule()["blk_warps"] == 8
