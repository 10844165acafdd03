"""chy_solve_static's work space holds one W array per solve: the largest grids that
its 8 MiB hold are solved, with chy_solve's bits, and the next larger are refused
with the bytes they need.  Collected last, like the entry point's other tests."""
import ctypes as C
import re

import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(96, 64, 64), (112, 32, 128)])
def test_fits(chylib, J, K, L):
    import torch
    plan = chylib.Plan(chylib.grid(J, K, L), "fp64", 1)
    for seed in (5, 6):
        rho = chylib.to_cuda_fortran(synth.disk_density(J, K, L, seed, spiral=True, spectrum=True))
        got = chylib.fortran_zeros_cuda(rho.shape)
        st = chylib.lib().chy_solve_static(plan._p, rho.data_ptr(), got.data_ptr(),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0, chylib.lib().chy_last_error()
        assert torch.equal(got, plan.solve(rho))


def test_refused_with_what_it_needs(chylib):
    plan = chylib.Plan(chylib.grid(128, 32, 128), "fp64", 1)
    buf = chylib.fortran_zeros_cuda(plan.shape)
    assert chylib.lib().chy_solve_static(plan._p, buf.data_ptr(), buf.data_ptr(), None) == 32   # CHY_ERR_CAPACITY
    need = int(re.search(rb"needs (\d+) bytes", chylib.lib().chy_last_error()).group(1))
    # X and W, and less than a quarter of them for moments and boundary sums
    two = 2 * 128 * 32 * 128 * 8
    assert two < need < 1.25 * two
