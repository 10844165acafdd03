"""A plan is ready on every stream when chy_plan_create returns: its tables formed on
the device, its work space cleared.  A solve on a stream that does not wait for the
default one, right behind the creation of a plan with a large work space (and
behind the iterate's allocation), gives the bits of a later one."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L,precision,n,corrections",
                         [(128, 64, 128, "fp64", 64, 1), (75, 64, 128, "mixed", 64, 1), (75, 64, 128, "mixed", 64, 2),
                          (257, 32, 64, "mixed", 64, 2), (66, 16, 64, "blktri", 64, 1)])
def test_solve_on_another_stream_at_once(chylib, J, K, L, precision, n, corrections):
    import torch
    rho = chylib.to_cuda_fortran(synth.disk_density(J, K, L, 8, spiral=True, spectrum=True))
    outs = [chylib.fortran_zeros_cuda(rho.shape) for _ in range(2)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    plan = chylib.Plan(chylib.grid(J, K, L), precision, n)
    plan.set_refine(corrections)
    plan.solve_batch([rho], [outs[0]], stream=s.cuda_stream)
    torch.cuda.synchronize()
    plan.solve_batch([rho], [outs[1]], stream=s.cuda_stream)
    torch.cuda.synchronize()
    assert float(outs[1].abs().max()) > 0.0 and torch.equal(outs[0], outs[1])
