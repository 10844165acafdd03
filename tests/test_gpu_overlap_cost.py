"""An FP64 solve whose sweeps keep their rows in device memory (JMAX > 257) is not
slowed by overlapped launches: one solve of 512x64x256, short enough to overlap,
costs little more than its share of a batch of two, which takes ordinary launches.
A single solve pays its launches and its last waves alone (a fifth at most), so
1.5 leaves room for noise."""
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


def test_single_solve_keeps_pace_with_a_batch(chylib):
    import torch
    J, K, L, n = 512, 64, 256, 6
    plan = chylib.Plan(chylib.grid(J, K, L), "fp64", 2)
    rho = chylib.to_cuda_fortran(synth.disk_density(J, K, L, 90, spiral=True, spectrum=True))
    outs = [chylib.fortran_zeros_cuda(plan.shape) for _ in range(2)]

    def time(count):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        best = float("inf")
        for _ in range(6):
            torch.cuda.synchronize()
            a.record()
            for _ in range(n):
                plan.solve_batch([rho] * count, outs[:count])
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) / (n * count))
        return best

    one, share = time(1), time(2)
    assert one < 1.5 * share, (one, share)
