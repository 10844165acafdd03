"""Mode solves of different kernels back to back on one stream, whose CTAs may be
resident side by side while they wait: every kernel that allocates tensor memory
(fused and wide mixed pipelines, FP64 sweeps, BLKTRI order) before and after every
other, launched directly and replayed from a graph, each solve bit for bit the
one that ran alone."""
import itertools

import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu

GRIDS = [(64, 32, 32, "mixed"), (65, 32, 32, "mixed"), (64, 32, 32, "fp64"), (66, 16, 32, "blktri")]


def test_every_order_of_the_mode_solves(chylib):
    import torch
    plans = [chylib.Plan(chylib.grid(J, K, L), prec, 1) for J, K, L, prec in GRIDS]
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 60 + i, spiral=True, spectrum=True))
            for i, (J, K, L, _) in enumerate(GRIDS)]
    ref = []
    for p, r in zip(plans, rhos):
        ref.append(p.solve(r))
        torch.cuda.synchronize()
    order = [i for pair in itertools.product(range(4), repeat=2) for i in pair]
    outs = [chylib.fortran_zeros_cuda(plans[i].shape) for i in order]

    def sequence():
        for i, f in zip(order, outs):
            plans[i].solve(rhos[i], f)

    def check():
        torch.cuda.synchronize()
        assert all(torch.equal(f, ref[i]) for i, f in zip(order, outs))
        for f in outs:
            f.zero_()

    for _ in range(3):
        sequence()
        check()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sequence()
    for _ in range(3):
        g.replay()
        check()
