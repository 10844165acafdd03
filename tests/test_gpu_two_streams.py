"""BLKTRI-order solves of two plans on two streams run side by side: the solves
queued on one stream do not hold the SMs that the other's need.  A solve of
128x64x128 takes 32 of the SMs, so a pair costs about one solve; a bound of 1.5
solves leaves room for both noise and a loaded host."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


def test_blktri_pairs_overlap(chylib):
    import torch
    J, K, L, n = 128, 64, 128, 6
    plans = [chylib.Plan(chylib.grid(J, K, L), "blktri", 1) for _ in range(2)]
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 80 + i, spiral=True, spectrum=True)) for i in range(2)]
    outs = [chylib.fortran_zeros_cuda(plans[0].shape) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]

    def run(which):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        main = torch.cuda.current_stream()
        torch.cuda.synchronize()
        a.record(main)
        for i in which:
            streams[i].wait_stream(main)
        for _ in range(n):
            for i in which:
                plans[i].solve_batch([rhos[i]], [outs[i]], stream=streams[i].cuda_stream)
        for i in which:
            main.wait_stream(streams[i])
        b.record(main)
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    run((0, 1))
    one = min(run((0,)) for _ in range(3))
    pair = min(run((0, 1)) for _ in range(3))
    assert pair < 1.5 * one, (pair / n, one / n)
