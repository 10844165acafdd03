"""The wide pipeline's radial sweeps around the row count that its rows in tensor
memory end at (M = JMAX - 1 = 512; 513 and more take the kernel with the rows in
device memory), with lower halves that fill their sixteen-row chunks and that do
not, and more items than SMs.

Tolerance: 1e-10 relative L2 over the write set against the oracle, the mixed
path's bar."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,K,L", [(290, 8, 32), (305, 32, 256), (449, 16, 32), (450, 16, 32), (512, 32, 64),
                                   (513, 16, 256), (514, 16, 32)])
def test_against_oracle(chylib, J, K, L):
    from oracle import oracle as O
    rho = synth.disk_density(J, K, L, 1100 + J, spiral=True, spectrum=True)
    ref = O.Oracle(J, K, L, nthreads=8).solve(rho)
    phi = np.zeros_like(rho, order="F")
    chylib.Plan(chylib.grid(J, K, L), "mixed", 1).solve(rho, phi)
    ws = (slice(0, J + 1), slice(0, K + 1))
    assert np.linalg.norm(phi[ws] - ref[ws]) < 1e-10 * np.linalg.norm(ref[ws])
