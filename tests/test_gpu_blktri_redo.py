"""BLKTRI-order passes that the tabulated pivots do not settle: with densities
scaled until every dividend lies below the range of the tabulated quotients, the
passes are formed again with divisions over the rows just stored, and the modes
are the host replay's bit for bit.  Partial solutions in tensor memory
(JMAX <= 257) and in shared memory."""
import ctypes as C

import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(66, 16, 64), (257, 8, 32), (258, 8, 32)])
def test_redone_passes_equal_host_replay(chylib, ora, J, K, L):
    M, NZ = J - 1, K - 1
    lib = chylib.lib()
    rho = synth.disk_density(J, K, L, 9, spiral=True, spectrum=True)
    g = chylib.grid(J, K, L)
    plan = chylib.Plan(g, "blktri", 1)
    plan.solve_batch([rho])
    usual = lib.chy_dbg_blk_redone()
    assert usual >= 0
    rho = np.asfortranarray(rho * 1e-265)
    plan.solve_batch([rho])
    assert lib.chy_dbg_blk_redone() > usual
    X = plan.debug_work("X", L * K * J).reshape(L, K, J)
    F = np.zeros((L, NZ, M))
    for k in range(NZ):
        for j in range(M):
            F[:, k, j] = ora.forward_real(rho[j + 1, k + 1, :].copy(), False)
    sc = np.zeros(8)
    assert lib.chy_dbg_table(C.byref(g), b"scalars", sc.ctypes.data_as(C.POINTER(C.c_double)), 8) == 8
    pig4, cmmax, cnmax = sc[1], sc[2], sc[4]
    assert np.any(X[:, :NZ, :M] != 0.0)
    for l in range(L):
        y = np.asfortranarray((pig4 * F[l]).T)
        y[:, NZ - 1] = y[:, NZ - 1] - cnmax * X[l, NZ, :M]
        y[M - 1, :] = y[M - 1, :] - cmmax * X[l, :NZ, M]
        assert lib.chy_dbg_blktri(C.byref(g), l, y.ctypes.data_as(C.POINTER(C.c_double))) == 0
        assert np.array_equal(y, X[l, :NZ, :M].T), l
