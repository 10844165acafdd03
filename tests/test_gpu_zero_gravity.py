"""GRAV = 0: no sources and a zero boundary, so PHI is zero in every precision
(the FP64 path divides the outer boundary's coefficient by 4 PI GRAV)."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed", "blktri"])
@pytest.mark.parametrize("J", [64, 65])
def test_phi_is_zero(chylib, precision, J):
    K, L = 16, 32
    rho = synth.disk_density(J, K, L, 3, spiral=True, spectrum=True)
    phi = chylib.Plan(chylib.grid(J, K, L, grav=0.0), precision, 1).solve(rho, np.full_like(rho, 7.0, order="F"))
    assert np.all(phi[:J + 1, :K + 1, :] == 0.0)
