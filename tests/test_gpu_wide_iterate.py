"""The wide mixed pipeline's FP64 iterate: only two or more corrections read it, so
only they allocate it (8 bytes a cell), and the solves with it are the same before
and after the first correction count that needs it."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


def test_allocated_on_demand(chylib):
    import torch
    J, K, L, n = 257, 16, 32, 2
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 20 + i, spiral=True, spectrum=True)) for i in range(n)]
    plan = chylib.Plan(chylib.grid(J, K, L), "mixed", n)
    base = plan.device_bytes
    one = plan.solve_batch(rhos)
    for c in (0, 1):
        plan.set_refine(c)
        assert plan.device_bytes == base
    plan.set_refine(2)
    assert plan.device_bytes == base + n * L * (K - 1) * J * 8
    two = plan.solve_batch(rhos)
    plan.set_refine(1)
    for a, b in zip(plan.solve_batch(rhos), one):
        assert torch.equal(a, b)
    other = chylib.Plan(chylib.grid(J, K, L), "mixed", n)
    other.set_refine(2)
    for a, b in zip(other.solve_batch(rhos), two):
        assert torch.equal(a, b) and not torch.equal(a, one[0])
