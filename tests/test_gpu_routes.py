"""Which kernels the sizes of a dispatch's edges run, asserted, and the kernels that
only plans without a pivot table reach.

The edges themselves are compared with the oracle and with one another in the
tests of each path; here the route is what is checked, so that a dispatch that
moves does not leave those tests without their subject."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu

ON_CHIP, OVERLAP = 1, 2


def density(chylib, J, K, L, seed):
    return chylib.to_cuda_fortran(synth.disk_density(J, K, L, seed, spiral=True, spectrum=True))


@pytest.mark.parametrize("J,K,L,precision,n,route",
                         # FP64 sweeps: rows in tensor memory up to M = 256, KMAX >= 32, until the groups of modes
                         # outnumber the SMs (KMAX = 128 with more than 128 rows: also beyond)
                         [(257, 32, 32, "fp64", 1, ON_CHIP), (258, 32, 32, "fp64", 1, 0), (64, 16, 32, "fp64", 1, 0),
                          (33, 32, 32, "fp64", 18, ON_CHIP), (33, 32, 32, "fp64", 20, 0),
                          (129, 128, 32, "fp64", 5, 0), (130, 128, 32, "fp64", 5, ON_CHIP),
                          # the wide pipeline's up to M = 512
                          (513, 16, 32, "mixed", 1, ON_CHIP), (514, 16, 32, "mixed", 1, 0)])
def test_sweeps(chylib, J, K, L, precision, n, route):
    plan = chylib.Plan(chylib.grid(J, K, L), precision, n)
    plan.solve_batch([density(chylib, J, K, L, 1)] * n)
    assert chylib.lib().chy_dbg_route(plan._p) & ON_CHIP == route


def test_overlap(chylib):
    """Launches overlap up to 9 M cells a launch sequence, one plan at a time."""
    lib = chylib.lib()
    J, K, L = 128, 64, 128                      # 1.04 M cells a solve
    a, b = (chylib.Plan(chylib.grid(J, K, L), "fp64", 9) for _ in range(2))
    rho = density(chylib, J, K, L, 2)
    for n, route in ((8, OVERLAP), (9, 0)):
        a.solve_batch([rho] * n)
        assert lib.chy_dbg_route(a._p) & OVERLAP == route
    chylib.solve_multi([a], [rho])
    assert lib.chy_dbg_route(a._p) & OVERLAP
    chylib.solve_multi([a, b], [rho, rho])
    assert not (lib.chy_dbg_route(a._p) | lib.chy_dbg_route(b._p)) & OVERLAP


@pytest.mark.parametrize("J,table", [(17, 0), (18, 1), (409, 1), (410, 0)])
def test_pivot_table_row_counts(chylib, J, table):
    """The fewest and the most rows that the tabulated kernel takes; the grids beyond
    them run the dividing one, and a declined table gives the same bits."""
    import torch
    K, L = 4, 32
    rho = density(chylib, J, K, L, 3)
    plan = chylib.Plan(chylib.grid(J, K, L), "blktri", 1)
    assert (plan.pivot_table_bytes > 0) == bool(table)
    bare = chylib.Plan(chylib.grid(J, K, L), "blktri", 1, pivot_table_max=0)
    assert bare.pivot_table_bytes == 0
    ref = plan.solve(rho)
    assert float(ref.abs().max()) > 0.0 and torch.equal(bare.solve(rho), ref)


@pytest.mark.parametrize("J,K,L,n", [(64, 32, 64, 2), (410, 8, 32, 1), (40, 8, 256, 20)])
def test_stage_schedules_of_the_dividing_kernel(chylib, J, K, L, n):
    """4, 8 and 16 warps a CTA, one CTA and more an SM: the tabulated kernel's bits
    (at 410 rows, where there is no table, the default schedule's)."""
    import torch
    rhos = [density(chylib, J, K, L, 30 + i) for i in range(n)]
    ref = chylib.Plan(chylib.grid(J, K, L), "blktri", n).solve_batch(rhos)
    plan = chylib.Plan(chylib.grid(J, K, L), "blktri", n, pivot_table_max=0)
    for nw, cps in ((8, 2), (4, 2), (4, 4), (8, 1), (16, 1)):
        plan.set_schedule(blk_warps=nw, blk_ctas_per_sm=cps)
        for a, b in zip(plan.solve_batch(rhos), ref):
            assert torch.equal(a, b), (nw, cps)


def test_edge_of_the_table_equals_host_replay(chylib, ora):
    """The largest grid with a table and the first without, mode by mode against the
    host replay of the recorded schedule."""
    import ctypes as C
    K, L = 4, 32
    for J in (409, 410):
        M, NZ = J - 1, K - 1
        rho = synth.disk_density(J, K, L, 9, spiral=True, spectrum=True)
        g = chylib.grid(J, K, L)
        plan = chylib.Plan(g, "blktri", 1)
        assert (plan.pivot_table_bytes > 0) == (J == 409)
        plan.solve_batch([rho])
        X = plan.debug_work("X", L * K * J).reshape(L, K, J)
        F = np.zeros((L, NZ, M))
        for k in range(NZ):
            for j in range(M):
                F[:, k, j] = ora.forward_real(rho[j + 1, k + 1, :].copy(), False)
        sc = np.zeros(8)
        dp = C.POINTER(C.c_double)
        assert chylib.lib().chy_dbg_table(C.byref(g), b"scalars", sc.ctypes.data_as(dp), 8) == 8
        for l in range(L):
            y = np.asfortranarray((sc[1] * F[l]).T)
            y[:, NZ - 1] = y[:, NZ - 1] - sc[4] * X[l, NZ, :M]
            y[M - 1, :] = y[M - 1, :] - sc[2] * X[l, :NZ, M]
            assert chylib.lib().chy_dbg_blktri(C.byref(g), l, y.ctypes.data_as(dp)) == 0
            assert np.array_equal(y, X[l, :NZ, :M].T), (J, l)
