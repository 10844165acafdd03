"""Short solves overlap their launches (programmatic stream serialization): the
same bits under CUDA graph capture, on a side stream behind the kernel that
writes RHO and before the one that overwrites it, and back to back on two
densities that share the plan's work arrays; a solve beyond the size limit takes
ordinary launches and agrees with itself alone."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L,prec", [(64, 32, 64, "fp64"), (64, 32, 64, "mixed"), (64, 32, 64, "blktri"),
                                        (257, 16, 64, "mixed"), (75, 16, 32, "mixed"), (75, 16, 32, "fp64")])
def test_capture_and_streams(chylib, J, K, L, prec):
    import torch
    a, b = (chylib.to_cuda_fortran(synth.disk_density(J, K, L, s, spiral=True, spectrum=True)) for s in (31, 32))
    plan = chylib.Plan(chylib.grid(J, K, L), prec, 1)
    ref = []
    for r in (a, b):
        ref.append(plan.solve(r))
        torch.cuda.synchronize()
    # back to back, alternating, no wait in between
    phis = [chylib.fortran_zeros_cuda(plan.shape) for _ in range(20)]
    for i, f in enumerate(phis):
        plan.solve((a, b)[i % 2], f)
    torch.cuda.synchronize()
    assert all(torch.equal(f, ref[i % 2]) for i, f in enumerate(phis))
    # a side stream: RHO written just before, overwritten just after
    s = torch.cuda.Stream()
    rho, out = torch.empty_like(a), chylib.fortran_zeros_cuda(plan.shape)
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for i in range(10):
            rho.copy_((a, b)[i % 2])
            plan.solve(rho, out)
            rho.fill_(float("nan"))
            phis[i].copy_(out)
    s.synchronize()
    assert all(torch.equal(phis[i], ref[i % 2]) for i in range(10))
    # captured and replayed
    rho.copy_(a)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.solve(rho, out)
    for r, want in ((b, ref[1]), (a, ref[0])):
        rho.copy_(r)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_beyond_the_limit(chylib):
    import torch
    J, K, L, n = 128, 128, 256, 3   # 13 M cells
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 40 + i, spiral=True, spectrum=True)) for i in range(n)]
    plan = chylib.Plan(chylib.grid(J, K, L), "fp64", n)
    for r, f in zip(rhos, plan.solve_batch(rhos)):
        assert torch.equal(plan.solve(r), f)
