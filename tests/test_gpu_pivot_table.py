"""The BLKTRI-order plan's pivot table as its caller sees it: how large it is, that
it can be declined, given back and made again with the same bits in PHI, that the
default does not depend on half of the device being free, and that a server makes
tables within its budget only."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu

J, K, L = 66, 16, 64


def test_declined_given_back_and_made_again(chylib):
    import torch
    rho = chylib.to_cuda_fortran(synth.disk_density(J, K, L, 5, spiral=True, spectrum=True))
    g = chylib.grid(J, K, L)
    plan = chylib.Plan(g, "blktri", 1)
    n = plan.pivot_table_bytes
    assert n > 0
    ref = plan.solve(rho)
    bare = chylib.Plan(g, "blktri", 1, pivot_table_max=0)
    assert bare.pivot_table_bytes == 0 and bare.device_bytes == plan.device_bytes - n
    assert torch.equal(bare.solve(rho), ref)
    for limit, have in ((n - 1, 0), (n, n), (0, 0), (-1, n), (n + 1, n)):
        plan.set_pivot_table(limit)
        assert plan.pivot_table_bytes == have and plan.device_bytes == bare.device_bytes + have
        assert torch.equal(plan.solve(rho), ref)


def test_only_blktri_plans_have_one(chylib):
    for precision in ("fp64", "mixed"):
        plan = chylib.Plan(chylib.grid(J, K, L), precision, 1, pivot_table_max=1 << 30)
        assert plan.pivot_table_bytes == 0
        with pytest.raises(chylib.ChyError) as e:
            plan.set_pivot_table(0)
        assert e.value.status == 10   # CHY_ERR_ARG


def test_default_with_less_than_half_the_device_free(chylib):
    import torch
    free, total = torch.cuda.mem_get_info()
    if free < 0.75 * total:
        pytest.skip("the device is in use")
    held = torch.empty(int(free - 0.4 * total), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 0.5 * total
        assert chylib.Plan(chylib.grid(J, K, L), "blktri", 1).pivot_table_bytes > 0
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.mark.parametrize("tables", [0, 1, 2])
def test_server_makes_tables_within_its_budget(chylib, tables):
    g = chylib.grid(J, K, L)
    plan = chylib.Plan(g, "blktri", 2)
    n, base = plan.pivot_table_bytes, plan.device_bytes - plan.pivot_table_bytes
    rho = synth.disk_density(J, K, L, 6, spiral=True, spectrum=True)
    ref = plan.solve(rho, np.zeros_like(rho, order="F"))
    plans = 2 * base + tables * n + n // 2      # the two lanes' plans, `tables` tables, no third half
    srv = chylib.Server("blktri", hbm_budget=2 * plans, max_batch=2, arena_fraction=0.5)
    try:
        phi = np.zeros_like(rho, order="F")
        srv.wait(srv.submit(g, rho, phi))
        assert np.array_equal(phi, ref)
        assert srv.stats()["plan_bytes"] == 2 * base + tables * n
    finally:
        srv.close()
