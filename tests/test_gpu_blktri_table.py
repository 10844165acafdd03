"""BLKTRI-order mode solve with tabulated pivots: bit for bit the host replay
of the recorded schedule (IEEE divisions) at the edges of its dispatch.

Rows M = JMAX-1 in whole chunks of eight and not, the fewest rows it takes, the
last row count whose partial solutions fit tensor memory and the first that
uses shared memory instead, the last with a table and the first without, one
and several warps per column set, and a grid long enough that solutions of
empty columns decay below the range of the tabulated quotients (the divisions'
path).  The disks' floor leaves exact zeros in most modes of the upper rows."""
import ctypes as C

import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(18, 4, 32), (24, 4, 32), (25, 8, 32), (65, 8, 64), (66, 16, 128), (257, 16, 32),
                                   (258, 16, 32), (380, 8, 32), (385, 4, 32), (386, 4, 32)])
def test_modes_equal_host_replay(chylib, ora, J, K, L):
    M, NZ = J - 1, K - 1
    rho = synth.disk_density(J, K, L, 9, spiral=True, spectrum=True)
    g = chylib.grid(J, K, L)
    plan = chylib.Plan(g, "blktri", 1)
    plan.solve_batch([rho])
    X = plan.debug_work("X", L * K * J).reshape(L, K, J)
    F = np.zeros((L, NZ, M))
    for k in range(NZ):
        for j in range(M):
            F[:, k, j] = ora.forward_real(rho[j + 1, k + 1, :].copy(), False)
    sc = np.zeros(8)
    assert chylib.lib().chy_dbg_table(C.byref(g), b"scalars", sc.ctypes.data_as(C.POINTER(C.c_double)), 8) == 8
    pig4, cmmax, cnmax = sc[1], sc[2], sc[4]
    for l in range(L):
        y = np.asfortranarray((pig4 * F[l]).T)
        y[:, NZ - 1] = y[:, NZ - 1] - cnmax * X[l, NZ, :M]
        y[M - 1, :] = y[M - 1, :] - cmmax * X[l, :NZ, M]
        assert chylib.lib().chy_dbg_blktri(C.byref(g), l, y.ctypes.data_as(C.POINTER(C.c_double))) == 0
        assert np.array_equal(y, X[l, :NZ, :M].T), l


def test_groups_beyond_the_sms(chylib):
    """More groups than SMs (several groups per CTA, no clusters) and one solve
    (clusters of eight) give the same bits."""
    import torch
    J, K, L, n = 40, 8, 256, 20
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 300 + i, spiral=True, spectrum=True)) for i in range(n)]
    batch = chylib.Plan(chylib.grid(J, K, L), "blktri", n).solve_batch(rhos)
    one = chylib.Plan(chylib.grid(J, K, L), "blktri", 1)
    for r, f in zip(rhos, batch):
        assert torch.equal(one.solve(r), f)
