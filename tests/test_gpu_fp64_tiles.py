"""FP64 eigenbasis mode solve at the edges of its tiles: odd JMAX (8-byte tile
copies), one row or column past a tile, the smallest KMAX, every KMAX variant,
and a batch large enough for the widest tiles against the single solves that
take the narrowest.

Tolerances: both solvers' errors grow like the operators' condition, the
square of the longer side, times 2^-53: the oracle's own BLKTRI solve is
2.4e-12 off at JMAX = 256, so 5e-12 there and 1e-12 up to a quarter of that
side.  Batch against single is bitwise: each value sums in an order that does
not depend on the tile width.
"""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(9, 4, 32), (33, 8, 32), (66, 16, 64), (65, 32, 64), (130, 32, 32), (257, 64, 32),
                                   (131, 128, 32)])
def test_against_oracle(chylib, J, K, L):
    from oracle import oracle as O
    rho = synth.disk_density(J, K, L, 100 + J, spiral=True, spectrum=True)
    ref = O.Oracle(J, K, L, nthreads=8).solve(rho)
    phi = np.zeros_like(rho, order="F")
    chylib.Plan(chylib.grid(J, K, L), "fp64", 1).solve(rho, phi)
    ws = (slice(0, J + 1), slice(0, K + 1))
    err = np.linalg.norm((phi[ws] - ref[ws]).ravel()) / np.linalg.norm(ref[ws].ravel())
    assert err < (1e-12 if J <= 66 else 5e-12), err


@pytest.mark.parametrize("J,K,L,n", [(66, 16, 64, 32), (67, 64, 64, 8), (96, 128, 128, 4)])
def test_tile_width_does_not_change_bits(chylib, J, K, L, n):
    import torch
    rhos = [chylib.to_cuda_fortran(synth.disk_density(J, K, L, 200 + i, spiral=True, spectrum=True)) for i in range(n)]
    batch = chylib.Plan(chylib.grid(J, K, L), "fp64", n).solve_batch(rhos)
    one = chylib.Plan(chylib.grid(J, K, L), "fp64", 1)
    for r, f in zip(rhos, batch):
        assert torch.equal(one.solve(r), f)
