"""A wait of the radial sweeps in tensor memory that runs out is reported: the FP64
path's k_thomas_tm and the wide mixed pipeline's k_wide_sweep_tm.  The hooks make
every CTA first wait on a barrier that nothing arrives on, with no copy issued, so
the failure path runs on purpose: NaN in PHI, CHY_ERR_TIMEOUT from the next call
that synchronises, and clean solves after it."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu

TIMEOUT = 31   # CHY_ERR_TIMEOUT


@pytest.mark.parametrize("J,K,L,precision", [(64, 32, 64, "fp64"), (130, 128, 32, "fp64"), (257, 16, 32, "mixed")])
def test_expired_wait_is_reported(chylib, J, K, L, precision):
    import torch
    lib = chylib.lib()
    probe = lib.chy_dbg_sweep_probe if precision == "fp64" else lib.chy_dbg_mixed_probe
    rho = synth.disk_density(J, K, L, 9, spiral=True, spectrum=True)
    rd = chylib.to_cuda_fortran(rho)
    plan = chylib.Plan(chylib.grid(J, K, L), precision, 2)

    def host():
        return plan.solve(rho, np.zeros_like(rho, order="F"))

    ref = host()
    assert np.all(np.isfinite(ref))
    try:
        assert probe(plan._p, 1000) == 0
        phi = np.zeros_like(rho, order="F")
        with pytest.raises(chylib.ChyError) as e:      # host pointers
            plan.solve(rho, phi)
        assert e.value.status == TIMEOUT and np.isnan(phi[1:J, 1:K, :]).all()
        with pytest.raises(chylib.ChyError) as e:      # device pointers with diagnostics
            plan.solve(rd, diag=True)
        assert e.value.status == TIMEOUT
        pd = plan.solve(rd)                            # asynchronous: the next call reports it
        torch.cuda.synchronize()
        assert torch.isnan(pd[1:J, 1:K, :]).all()
        assert probe(plan._p, 0) == 0
        with pytest.raises(chylib.ChyError) as e:
            host()
        assert e.value.status == TIMEOUT
    finally:
        probe(plan._p, 0)
    assert np.array_equal(host(), ref)
    out, _ = plan.solve(rd, diag=True)
    assert np.array_equal(out.cpu().numpy(), ref)


def test_probe_needs_an_fp64_plan(chylib):
    plan = chylib.Plan(chylib.grid(64, 32, 64), "mixed", 1)
    assert chylib.lib().chy_dbg_sweep_probe(plan._p, 10) == 10   # CHY_ERR_ARG
