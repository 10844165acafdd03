"""The azimuthal transforms at every LMAX and at JMAX one column short of, at
and past the widths of their tiles (8, 16 and 32 columns; an odd JMAX takes the
8-byte copies, an even one the tensor maps).

Tolerance: 2e-12 relative L2 over the write set against the oracle, the FP64
path's bar on every other grid; a column read or written in the wrong place, or
a twiddle of the wrong stage, is an error of order one in that column."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("J", [17, 24, 31, 34])
def test_every_lmax(chylib, J, L):
    from oracle import oracle as O
    K = 8
    rho = synth.disk_density(J, K, L, 800 + J, spiral=True, spectrum=True)
    ref = O.Oracle(J, K, L, nthreads=8).solve(rho)
    phi = np.zeros_like(rho, order="F")
    chylib.Plan(chylib.grid(J, K, L), "fp64", 1).solve(rho, phi)
    for j in range(J + 1):                       # column by column: one bad column shows
        a, b = phi[j, :K + 1], ref[j, :K + 1]
        assert np.linalg.norm(a - b) < 2e-12 * np.linalg.norm(b), j
