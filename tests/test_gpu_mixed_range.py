"""Mixed solves whose modes span a wide range: compact bodies without a density
floor, whose tails run through every magnitude down to zero, so that a tile or a
radial half holds nothing but values whose power-of-two scale leaves single
precision; and densities that are small as a whole.

Tolerance: the mixed path's 1e-10 against the FP64 path, relative L2 over the write
set; at 1e-25 of a unit density, where the correction's residual falls below
single precision's range, 1e-8; at 1e-30 no more than finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def body(J, K, L, sigma, r0=0.0):
    """A Gaussian body of width sigma around (r0, 0), m = 2 and 5 parts, no floor."""
    r, z = (np.arange(J) + 0.5) / J, (np.arange(K) + 0.5) * 0.5 / K
    psi = (np.arange(L) + 0.5) * 2.0 * np.pi / L
    a = np.zeros((J + 2, K + 2, L), order="F")
    g = np.exp(-((r[:, None] - r0) ** 2 + z[None, :] ** 2) / sigma ** 2)
    a[1:J + 1, 1:K + 1, :] = g[:, :, None] * (1.0 + 0.3 * np.cos(2.0 * psi) + 0.1 * np.cos(5.0 * psi))
    return a


def error(chylib, rho, J, K, L, kernel=0, **kw):
    g = chylib.grid(J, K, L, **kw)
    ref = chylib.Plan(g, "fp64", 1).solve(rho, np.zeros_like(rho, order="F"))
    plan = chylib.Plan(g, "mixed", 1)
    plan.set_schedule(mode_kernel=kernel)
    got = plan.solve(rho, np.zeros_like(rho, order="F"))
    ws = (slice(0, J + 1), slice(0, K + 1))
    big = np.abs(ref[ws]).max()
    return float(np.linalg.norm((got - ref)[ws] / big) / np.linalg.norm(ref[ws] / big))


SIGMAS = [0.1, 0.06, 0.055, 0.05, 0.045, 0.04, 0.035, 0.03, 0.025, 0.02, 0.015]


@pytest.mark.parametrize("J,K,L", [(257, 32, 32), (300, 16, 32), (145, 16, 32), (513, 16, 32)])
@pytest.mark.parametrize("maxtrm", [10, 0])
def test_compact_bodies_wide(chylib, J, K, L, maxtrm):
    for sigma in SIGMAS:
        for r0 in (0.0, 0.9):
            e = error(chylib, body(J, K, L, sigma, r0), J, K, L, literal="r8", maxtrm=maxtrm)
            assert e < 1e-10, (sigma, r0, e)


@pytest.mark.parametrize("J,K,L", [(127, 32, 32), (250, 16, 32), (256, 16, 32)])
@pytest.mark.parametrize("maxtrm", [10, 0])
@pytest.mark.parametrize("kernel", [1, 2])
def test_compact_bodies_fused(chylib, J, K, L, maxtrm, kernel):
    for sigma in SIGMAS:
        for r0 in (0.0, 0.9):
            e = error(chylib, body(J, K, L, sigma, r0), J, K, L, kernel, literal="r8", maxtrm=maxtrm)
            assert e < 1e-10, (sigma, r0, e)


@pytest.mark.parametrize("J,K,L", [(71, 8, 64), (81, 8, 64), (128, 16, 32), (257, 16, 32)])
def test_small_densities(chylib, J, K, L):
    from chymera_uo_b200 import synth
    rho = synth.disk_density(J, K, L, 5, spiral=True, spectrum=True)
    for scale, tol in ((1e30, 1e-10), (1e-20, 1e-10), (1e-25, 1e-8), (1e-30, np.inf)):
        e = error(chylib, np.asfortranarray(rho * scale), J, K, L)
        assert np.isfinite(e) and e < tol, (scale, e)


@pytest.mark.parametrize("J,K,L", [(127, 32, 32), (128, 32, 32), (257, 16, 32)])
def test_centimetres_and_grams(chylib, J, K, L):
    """The same bodies in units in which lengths are 1e13 and the right-hand side 1e-15:
    the solution is 2^86 times the residual."""
    for sigma, r0 in ((0.2, 0.0), (0.05, 0.0), (0.05, 0.9), (0.02, 0.0)):
        e = error(chylib, body(J, K, L, sigma, r0) * 1e-9, J, K, L, rof3n=1e13 / J, zof3n=0.5e13 / K, grav=6.67e-8)
        assert e < 1e-10, (sigma, r0, e)
