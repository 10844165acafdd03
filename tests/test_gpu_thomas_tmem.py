"""The FP64 path's radial sweeps with the rows in tensor memory against the kernel
with the rows in device memory, which serves the same grids once their groups of
modes outnumber the SMs (and KMAX = 128 with at most 128 rows): the recurrences
are the same, so a batch of the one equals single solves of the other bit for
bit.  Row counts M = JMAX - 1 at the edges of the sixteen-row chunks and at the
largest (256; 257 takes the kernel with the rows in device memory both times)."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu

EDGES = [16, 17, 18, 33, 100, 129]


@pytest.mark.parametrize("J,K", [(J, K) for K in (32, 64, 128) for J in EDGES]
                         + [(J, K) for K in (32, 64) for J in (130, 242, 256, 257, 258)])
def test_both_kernels_agree_bitwise(chylib, J, K):
    import torch
    L = 32
    groups = L * K // 128
    n = 160 // groups                      # 160 groups: more than the SMs
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 950 + i, spiral=True, spectrum=True)) for i in range(2)]
    batch = chylib.Plan(chylib.grid(J, K, L), "fp64", n).solve_batch([rhos[i % 2] for i in range(n)])
    one = chylib.Plan(chylib.grid(J, K, L), "fp64", 1)
    single = [one.solve(r) for r in rhos]
    assert float(single[0].abs().max()) > 0.0
    for i, f in enumerate(batch):
        assert torch.equal(single[i % 2], f), i


@pytest.mark.parametrize("J,L,n", [(200, 64, 5), (140, 32, 11)])
def test_many_groups_per_sm(chylib, J, L, n):
    """KMAX = 128 and more than 128 rows: several groups through one CTA's slots."""
    import torch
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, 128, L, 970 + i, spiral=True, spectrum=True)) for i in range(n)]
    batch = chylib.Plan(chylib.grid(J, 128, L), "fp64", n).solve_batch(rhos)
    one = chylib.Plan(chylib.grid(J, 128, L), "fp64", 1)
    for r, f in zip(rhos, batch):
        assert torch.equal(one.solve(r), f)
