"""ZAXPHI's extrapolation on the GPU for every NPOINT and several LMAX: the row
PHI(JMAX+2, K, :) equals pot/pot3.f:334-378 evaluated in numpy's IEEE double
arithmetic on the returned PHI, bit for bit, and PHICHK / KLOCAT follow from it.
A zero density (zero potentials) takes the dividing path."""
import numpy as np
import pytest

from chymera_uo_b200 import synth

pytestmark = pytest.mark.gpu


def zaxphi(phi, J, K, L, npoint, rhf):
    lm, ichk = L // 2, npoint % 2
    num = (npoint - ichk) // 2
    x = np.zeros(npoint + 1)
    for j in range(2, num + 2):
        x[num + (j - 1)], x[num - (j - 2)] = rhf[j - 1], -rhf[j - 1]
    if ichk:
        x[2 * num + 1] = rhf[num + 1]
    p = np.zeros((npoint + 1, K, lm))
    for j in range(2, num + 2):
        p[num + (j - 1)], p[num - (j - 2)] = phi[j - 1, 1:K + 1, :lm], phi[j - 1, 1:K + 1, lm:]
    if ichk:
        p[2 * num + 1] = phi[num + 1, 1:K + 1, :lm]
    for i in range(1, npoint):
        p1, xinv = p[i].copy(), 1.0 / x[i]
        xr = 0.0 * xinv
        for j in range(i + 1, npoint + 1):
            xratio = x[j] * xinv
            p[j] = (p1 * (xratio - xr) + p[j] * (xr - 1.0)) / (xratio - 1.0)
    return p[npoint]


@pytest.mark.parametrize("npoint", range(2, 11))
@pytest.mark.parametrize("L", [32, 64, 256])
def test_axis_row(chylib, npoint, L):
    J, K = 24, 8
    rho = synth.disk_density(J, K, L, 70 + npoint, spiral=True, spectrum=True)
    phi = np.zeros_like(rho, order="F")
    _, (d,) = chylib.Plan(chylib.grid(J, K, L, npoint=npoint), "fp64", 1).solve_batch([rho], [phi], diag=True)
    ref = zaxphi(phi, J, K, L, npoint, synth.default_grid(J, K, L).rhf())
    assert np.array_equal(phi[J + 1, 1:K + 1, :L // 2], ref)
    assert np.array_equal(phi[J + 1, 1:K + 1, L // 2:], ref)
    er = 1.0 - ref / ref[np.arange(K), np.abs(ref).argmax(1)][:, None]
    phac = er[np.arange(K), np.abs(er).argmax(1)]
    assert d["klocat"] == int(np.abs(phac).argmax()) + 2 and d["phichk"] == phac[d["klocat"] - 2]


def test_zero_density(chylib):
    J, K, L = 24, 8, 32
    rho = np.zeros((J + 2, K + 2, L), order="F")
    phi = np.ones_like(rho, order="F")
    chylib.Plan(chylib.grid(J, K, L), "fp64", 1).solve_batch([rho], [phi])
    assert np.all(phi[:J + 1, :K + 1] == 0.0) and np.all(phi[J + 1, 1:K + 1] == 0.0)
