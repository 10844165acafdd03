"""The wide mixed pipeline at the edges of its 64-column tiles and its two-sided
sweeps: JMAX = 1 mod 16 up to 256 (the last column of a tile, of a half, alone in
a tile), odd and even JMAX above 256, small and large KMAX, no, one, two and
three corrections (each source and destination of the iterate).

Tolerance: 1e-10 relative L2 over the write set against the oracle after one
correction, 1e-11 after two or more (the oracle's own accuracy), 1e-4 without one
(FP32 sweeps), as for the other mixed grids; a batch equals its singles bitwise."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(65, 8, 32), (129, 32, 32), (241, 16, 64), (257, 32, 32), (258, 4, 32), (319, 64, 32),
                                   (321, 128, 32), (385, 16, 32), (1023, 8, 32)])
def test_against_oracle(chylib, J, K, L):
    from oracle import oracle as O
    rho = synth.disk_density(J, K, L, 600 + J, spiral=True, spectrum=True)
    ref = O.Oracle(J, K, L, nthreads=8).solve(rho)
    ws = (slice(0, J + 1), slice(0, K + 1))
    plan = chylib.Plan(chylib.grid(J, K, L), "mixed", 1)
    for corrections, tol in ((0, 1e-4), (1, 1e-10), (2, 1e-11), (3, 1e-11)):
        plan.set_refine(corrections)
        phi = np.zeros_like(rho, order="F")
        _, (d,) = plan.solve_batch([rho], [phi], diag=True)
        assert chylib.lib().chy_dbg_mixed_kernel(plan._p) == 3
        err = np.linalg.norm((phi[ws] - ref[ws]).ravel()) / np.linalg.norm(ref[ws].ravel())
        assert err < tol, (corrections, err)
        assert d["iterations"] == corrections + 1 and d["corr_rel"][0] == pytest.approx(1.0)
        assert corrections == 0 or d["corr_rel"][1] < 1e-4
        assert np.all(phi[:, K + 1, :] == 0.0) and np.all(phi[J + 1, 0, :] == 0.0)


@pytest.mark.parametrize("J,K,L,n", [(241, 32, 64, 9), (450, 16, 128, 5)])
def test_batch_equals_singles(chylib, J, K, L, n):
    import torch
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 700 + i, spiral=True, spectrum=True)) for i in range(n)]
    batch = chylib.Plan(chylib.grid(J, K, L), "mixed", n).solve_batch(rhos)
    one = chylib.Plan(chylib.grid(J, K, L), "mixed", 1)
    for r, f in zip(rhos, batch):
        assert torch.equal(one.solve(r), f)
