"""Mixed plans whose JMAX is not a multiple of 16: rows of X padded to whole
16-column tiles for the fused mode solve (kernel 1 or 2), JMAX = 1 mod 16 by the
wide pipeline (kernel 3).  One column past and short of a tile, of a 32-column
chunk and of a 64-column half; small KMAX and the largest.

Tolerance: 1e-10 relative L2 over the write set against the oracle, the mixed
path's bar; two corrections 1e-11 (the oracle's own accuracy, as on the other
grids)."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("J,K,L,isym", [(66, 16, 32, 2), (79, 32, 64, 1), (95, 32, 64, 2), (98, 64, 32, 2),
                                        (130, 8, 64, 2), (189, 64, 64, 1), (194, 32, 32, 2), (255, 128, 32, 2),
                                        (65, 32, 32, 2), (193, 16, 32, 2)])
def test_against_oracle(chylib, J, K, L, isym):
    from oracle import oracle as O
    rho = synth.disk_density(J, K, L, 400 + J, spiral=True, spectrum=True)
    ref = O.Oracle(J, K, L, nthreads=8).solve(rho, isym=isym)
    ws = (slice(0, J + 1), slice(0, K + 1))
    plan = chylib.Plan(chylib.grid(J, K, L, isym=isym), "mixed", 1)
    for corrections, tol in ((1, 1e-10), (2, 1e-11)):
        plan.set_refine(corrections)
        phi = np.zeros_like(rho, order="F")
        plan.solve(rho, phi)
        assert chylib.lib().chy_dbg_mixed_kernel(plan._p) == (3 if J % 16 == 1 else 1)
        assert rel_l2(phi[ws], ref[ws]) < tol, corrections
        assert np.all(phi[:, K + 1, :] == 0.0) and np.all(phi[J + 1, 0, :] == 0.0)


@pytest.mark.parametrize("J,K,L,n", [(72, 32, 64, 40), (189, 64, 128, 20), (250, 128, 256, 12)])
def test_pairs_batches_and_singles_agree_bitwise(chylib, J, K, L, n):
    import torch
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 500 + i, spiral=True, spectrum=True)) for i in range(n)]
    plan = chylib.Plan(chylib.grid(J, K, L), "mixed", n)
    batch = plan.solve_batch(rhos)
    assert chylib.lib().chy_dbg_mixed_kernel(plan._p) == 2
    one = chylib.Plan(chylib.grid(J, K, L), "mixed", 1)
    for r, f in zip(rhos, batch):
        assert torch.equal(one.solve(r), f)
    assert chylib.lib().chy_dbg_mixed_kernel(one._p) == 1


def test_coef_output(chylib):
    """/COEFS/ reads X by its padded rows: the same values as the FP64 plan's,
    whose transform is the same."""
    import torch
    J, K, L = 75, 16, 32
    rho = chylib.to_cuda_fortran(synth.disk_density(J, K, L, 7, spiral=True, spectrum=True))
    out = []
    for prec in ("fp64", "mixed"):
        plan = chylib.Plan(chylib.grid(J, K, L), prec, 1)
        coef = torch.zeros((2, L // 2, K + 2, J + 2), dtype=torch.float64, device="cuda")
        plan.set_coef(coef)
        plan.solve(rho)
        out.append(coef)
    assert torch.equal(out[0], out[1])
