"""Timed cases of the gravitational-potential solve.

Each case is work a simulation code or a post-processing job hands to this
library through its public Python entry points (``Plan``, ``solve_multi``):
seeded self-gravitating disks (flared base disk, m = 2 spiral, m <= 32
spectrum, cell noise, as the repository's synthetic workloads) on grids of the
sizes that its tests and its benchmark use, and on sizes between them.

A case is a dict:

* ``kind``: ``solve`` (device arrays, one grid), ``host`` (pinned host arrays
  through the same call), ``multi`` (grids of several sizes in one call),
  ``step`` (a time step's gravity: solve with the star's potential, then the
  momentum source terms);
* ``jmax``, ``kmax``, ``lmax``: the grid; KMAX and LMAX are powers of two (the
  method's rule), JMAX is any number;
* ``n``: densities per call;
* ``precision``: ``mixed``, ``fp64`` or ``blktri``;
* ``literal``: transform constants as a default build or a promoted-literal
  (``r8``) build of the reference has them;
* ``isym``: BDYGEN's symmetry flag (2: mirror symmetry about the midplane, the
  production value; 1: none).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import chymera_uo_b200 as chy

PI = 3.1415926535897932

# grids of the `multi` kind: the size set of the batched workload
MULTI_J, MULTI_K, MULTI_L = (64, 128, 256), (32, 64, 128), (64, 128, 256)


def _case(name, kind, j, k, l, n, precision, literal="gcc", isym=2):
    return {"name": name, "kind": kind, "jmax": j, "kmax": k, "lmax": l, "n": n, "precision": precision,
            "literal": literal, "isym": isym}


def listed():
    return [
        # the size of the reference's CPU runs, one density at a time, as a
        # time-step loop calls it: launches and latency count
        _case("small_fp64", "solve", 64, 32, 64, 1, "fp64", "r8"),
        _case("small_mixed", "solve", 64, 32, 64, 1, "mixed"),
        # the same grid through the reference's own cyclic reduction (the
        # setting for runs that have to follow the reference's rounding)
        _case("small_blktri", "solve", 64, 32, 64, 1, "blktri"),
        # the production grid, one density per time step
        _case("large_mixed", "solve", 256, 128, 256, 1, "mixed", "r8"),
        _case("large_blktri", "solve", 256, 128, 256, 1, "blktri"),
        # an ensemble or a stack of snapshots on the production grid: the
        # benchmark's default workload, and a smaller stack in FP64
        _case("batch_mixed", "solve", 256, 128, 256, 32, "mixed"),
        _case("batch_fp64", "solve", 256, 128, 256, 8, "fp64", "r8"),
        # the largest grid that the benchmark serves
        _case("wide_mixed", "solve", 512, 128, 512, 4, "mixed", "r8"),
        # a grid whose radius was cut at an odd zone count, no mirror symmetry
        _case("odd_mixed", "solve", 189, 64, 128, 4, "mixed", "r8", isym=1),
        # a parameter study: 24 disks on grids of uneven sizes in one call
        _case("uneven_mixed", "multi", 256, 128, 256, 24, "mixed"),
        # one time step's gravity: solve, star and indirect term, source terms
        _case("step_mixed", "step", 256, 128, 256, 1, "mixed"),
        # densities that live in host memory (a Fortran or numpy caller)
        _case("host_mixed", "host", 256, 128, 256, 6, "mixed", "r8"),
    ]


def draw(rng):
    while True:
        kind = rng.choice(["solve"] * 7 + ["host", "multi", "step"])
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64", "fp64", "blktri"])
        lo = 64 if precision == "mixed" else 32
        j = int(round(math.exp(rng.uniform(math.log(lo), math.log(512)))))
        k = rng.choice([16, 32, 64, 128])
        l = rng.choice([32, 64, 128, 256, 512])
        n = int(round(math.exp(rng.uniform(0.0, math.log(32)))))
        if kind == "multi":
            precision = rng.choice(["mixed", "fp64"])
            j, k, l = MULTI_J[-1], MULTI_K[-1], MULTI_L[-1]
        elif kind == "step":
            n = 1
        elif kind == "host":
            n = min(n, 6)
        cells = n * j * k * l
        cap = {"mixed": 32, "fp64": 16, "blktri": 4}[precision] * 256 * 128 * 256
        if kind == "host":
            cap = 6 * 256 * 128 * 256
        if cells > cap or (precision == "blktri" and j * k > 256 * 128):
            continue
        c = _case("", kind, j, k, l, n, precision, rng.choice(["gcc", "r8"]), rng.choice([2, 2, 1]))
        del c["name"]
        return c


def _sizes(case):
    """(jmax, kmax, lmax) of every density of a case."""
    if case["kind"] != "multi":
        return [(case["jmax"], case["kmax"], case["lmax"])] * case["n"]
    # the whole size set in a fixed scattered order
    return [(MULTI_J[(i * 2) % 3], MULTI_K[(i // 3 + i) % 3], MULTI_L[(i // 9 + 2 * i) % 3]) for i in range(case["n"])]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _noise(n, seed, device):
    """n values in [-1, 1): a hash of the index, the same on every device."""
    h = torch.arange(n, dtype=torch.int64, device=device) * 2654435761 + (seed * 40503 + 12345)
    for mul, sh in ((0x9E3779B1, 15), (0x85EBCA6B, 13), (0xC2B2AE35, 16)):
        h = (h & 0x7FFFFFFF) * mul
        h = h ^ (h >> sh)
    return (h & 0xFFFFFF).to(torch.float64) / float(1 << 23) - 1.0


def _density(j, k, l, seed, device):
    """RHO(JMAX+2, KMAX+2, LMAX), column-major: a flared disk with random
    slope and scale height, spiral, azimuthal spectrum and cell noise."""
    r = np.random.default_rng(seed)
    slope, h, phases = r.uniform(-2.0, -1.0), r.uniform(0.03, 0.1), r.uniform(0.0, 2.0 * PI, 32)
    rhf = (torch.arange(j, dtype=torch.float64, device=device) + 0.5) / j
    zhf = (torch.arange(k, dtype=torch.float64, device=device) + 0.5) * (0.5 / k)
    psi = (torch.arange(l, dtype=torch.float64, device=device) + 0.5) * (2.0 * PI / l)
    r_out = (j - 1) / j
    sig = (rhf / r_out) ** slope * torch.exp(-((rhf / (0.8 * r_out)) ** 4))
    hh = h * rhf
    base = (sig / (math.sqrt(2.0 * PI) * hh))[None, :] * torch.exp(-(zhf[:, None] ** 2) / (2.0 * hh[None, :] ** 2))
    spiral = 1.0 + 0.05 * torch.cos(2.0 * (psi[:, None] - torch.log(rhf / r_out)[None, :] / math.tan(math.radians(15.0))))
    m = torch.arange(1, 33, dtype=torch.float64, device=device)
    ph = torch.from_numpy(phases).to(device)
    spec = 1.0 + (0.02 * m ** -2 * torch.cos(m * psi[:, None] + ph)).sum(1)
    rho = base[None] * (spiral * spec[:, None])[:, None, :]                  # [l][k][j]
    rho = rho * (1.0 + 1e-3 * _noise(l * k * j, seed, device).reshape(l, k, j))
    rho = torch.maximum(rho, 1e-10 * rho.max())
    out = torch.zeros((l, k + 2, j + 2), dtype=torch.float64, device=device)
    out[:, 1:k + 1, 1:j + 1] = rho
    return out.permute(2, 1, 0)


def _pinned(shape):
    return torch.zeros(shape[::-1], dtype=torch.float64).pin_memory().numpy().transpose()


def prepare(case, seed):
    dev = torch.device("cuda")
    sizes = _sizes(case)
    plans = {}
    for size in sizes:
        if size not in plans:
            batch = sum(s == size for s in sizes)
            g = chy.grid(*size, literal=case["literal"], isym=case["isym"])
            plans[size] = chy.Plan(g, case["precision"], max_batch=1 if case["kind"] == "host" else batch)
    rhos = [_density(*size, 64 * seed + i, dev) for i, size in enumerate(sizes)]
    state = {"kind": case["kind"], "plans": [plans[s] for s in sizes]}
    if case["kind"] == "host":
        state["phis"] = [_pinned(tuple(r.shape)) for r in rhos]
        state["rhos"] = [_pinned(tuple(r.shape)) for r in rhos]
        for h, r in zip(state["rhos"], rhos):
            h[...] = r.cpu().numpy()
        return state
    state["rhos"], state["phis"] = rhos, [chy.fortran_zeros_cuda(tuple(r.shape)) for r in rhos]
    if case["kind"] == "step":
        rho = rhos[0]
        state["plans"][0].set_external(1.0, tmassacc=0.01, rpstar=0.02, phi_star=0.7, indirect=True)
        rhf = (torch.arange(rho.shape[0], dtype=torch.float64, device=dev) - 0.5) / case["jmax"]
        omega = chy.fortran_zeros_cuda(tuple(rho.shape))
        omega += (rhf.abs() + 0.05)[:, None, None] ** -1.5
        pressure = chy.fortran_zeros_cuda(tuple(rho.shape))
        pressure += 1e-3 * rho.abs() ** (5.0 / 3.0)
        state["hydro"] = (omega, pressure)
        # momentum densities, updated in place step after step
        state["sta"] = [chy.fortran_zeros_cuda(tuple(rho.shape)) for _ in range(3)]
    return state


def run(state):
    plans, rhos, phis = state["plans"], state["rhos"], state["phis"]
    if state["kind"] == "multi":
        return chy.solve_multi(plans, rhos, phis)
    plans[0].solve_batch(rhos, phis)
    if state["kind"] == "step":
        omega, p = state["hydro"]
        s, t, a = state["sta"]
        plans[0].source(rhos[0], phis[0], omega, p, s, t, a, delt=1e-4)
        return {"phi": phis[0], "s": s, "t": t, "a": a}
    return phis


def work(case):
    """RHO in and PHI out once (and for a step OMEGA, P in, S, T, A in and
    out); operations of a direct solver with fast transforms."""
    nbytes = flops = 0.0
    for j, k, l in _sizes(case):
        cells = float((j + 2) * (k + 2) * l)
        nbytes += 16.0 * cells
        # two transforms each along the azimuth and the height, one
        # elimination along the radius
        flops += j * k * l * (2 * 2.5 * math.log2(l) + 2 * 2.5 * math.log2(k) + 8.0)
        if case["kind"] == "step":
            nbytes += 8.0 * 8.0 * cells
            flops += 40.0 * j * k * l
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The solution in 64 bits, by a dense eigenbasis along the height and
# elimination along the radius, with the boundary from normalised multipoles
# ---------------------------------------------------------------------------
def _legendre(lmax, m, x):
    """P_l^m(x) for l = m..lmax, without the (-1)^m phase."""
    s = torch.sqrt(1.0 - x * x)
    p = [torch.ones_like(x)]
    for i in range(m):
        p[0] = p[0] * (2 * i + 1) * s
    if lmax > m:
        p.append((2 * m + 1) * x * p[0])
    for l in range(m + 2, lmax + 1):
        p.append(((2 * l - 1) * x * p[-1] - (l + m - 1) * p[-2]) / (l - m))
    return p


def _boundary(rho, j, k, l, isym, rhf, zhf, psi):
    """Potential at the top edge (rhf[1..j], zhf[k]) and the outer edge
    (rhf[j], zhf[1..k-1]), [points][l]; rho: [l][k-1][j-1]."""
    maxtrm, dth, dz, dr = 10, 2.0 * PI / l, 0.5 / k, 1.0 / j
    f2 = 2.0 if isym == 2 else 1.0
    zz, rr = zhf[1:k][:, None], rhf[1:j][None, :]
    rs = torch.sqrt(rr * rr + zz * zz)
    dv = 0.5 * dth * dz * ((rr + 0.5 * dr) ** 2 - (rr - 0.5 * dr) ** 2) * f2 + 0.0 * rs
    order = torch.argsort(rs.reshape(-1), stable=True)
    rsort, cs = rs.reshape(-1)[order], (zz / rs).reshape(-1)[order]
    rb = torch.cat([torch.sqrt(zhf[k] ** 2 + rhf[1:j + 1] ** 2), torch.sqrt(rhf[j] ** 2 + zhf[1:k] ** 2)])
    cb = torch.cat([zhf[k] / rb[:j], zhf[1:k] / rb[j:]])
    at = torch.searchsorted(rsort, rb, right=True)
    zero = torch.zeros(1, dtype=torch.float64, device=rho.device)
    phi = torch.zeros((rb.numel(), l), dtype=torch.float64, device=rho.device)
    flat = rho.reshape(l, -1)
    for m in range(maxtrm + 1):
        p, pb = _legendre(maxtrm, m, cs), _legendre(maxtrm, m, cb)
        for part in ((torch.cos(m * psi),) if m == 0 else (torch.cos(m * psi), torch.sin(m * psi))):
            mom = (part @ flat * dv.reshape(-1))[order]
            total = torch.zeros_like(rb)
            for n in range(m, maxtrm + 1):
                if isym == 2 and (n + m) % 2:
                    continue
                q = p[n - m] * mom
                inner = torch.cat([zero, torch.cumsum(q * rsort ** n, 0)])[at]
                outer = torch.cat([torch.flip(torch.cumsum(torch.flip(q * rsort ** (-n - 1), [0]), 0), [0]), zero])[at]
                norm = (1.0 if m == 0 else 2.0) * math.factorial(n - m) / math.factorial(n + m)
                total = total + norm * pb[n - m] * (inner * rb ** (-n - 1) + outer * rb ** n)
            phi -= total[:, None] * part[None, :]
    return phi


def _axis_value(phi, j, l, rhf):
    """PHI on the axis: the interpolating polynomial of eight points through
    the axis, at radius 0; phi: [l][k][j], radii rhf[1..]."""
    num = 4
    x = torch.cat([-rhf[1:num + 1].flip(0), rhf[1:num + 1]])
    w = torch.ones_like(x)
    for a in range(2 * num):
        for b in range(2 * num):
            if a != b:
                w[a] = w[a] * x[b] / (x[b] - x[a])
    half = l // 2
    v = torch.cat([phi[half:, :, :num].flip(2), phi[:half, :, :num]], 2) @ w
    return torch.cat([v, v], 0)


def _solve(rho_full, j, k, l, isym):
    dev, f8 = rho_full.device, torch.float64
    dr, dz, dth = 1.0 / j, 0.5 / k, 2.0 * PI / l
    rhf = (torch.arange(j + 2, dtype=f8, device=dev) - 0.5) * dr          # rhf[i] is RHF(i+1)
    zhf = (torch.arange(k + 2, dtype=f8, device=dev) - 0.5) * dz
    psi = (torch.arange(l, dtype=f8, device=dev) + 0.5) * dth
    rho = rho_full.permute(2, 1, 0)[:, 1:k, 1:j]                          # [l][k-1][j-1]
    bdy = _boundary(rho, j, k, l, isym, rhf, zhf, psi)
    m_, nz = j - 1, k - 1
    r = rhf[1:j]
    c = (1.0 / dr + 0.5 / r) / dr
    a = (1.0 / dr - 0.5 / r) / dr
    cc = 1.0 / (r * dth) ** 2
    y = 4.0 * PI * torch.fft.rfft(rho, dim=0)                              # [mode][k][j]
    b = torch.fft.rfft(bdy, dim=1)
    y[:, nz - 1, :] -= b[:m_].T / (dz * dz)
    y[:, :, m_ - 1] -= b[j:].T * c[m_ - 1]
    tz = torch.zeros((nz, nz), dtype=f8, device=dev)
    i = torch.arange(nz, device=dev)
    tz[i, i] = -2.0 / (dz * dz)
    tz[0, 0] = -1.0 / (dz * dz)
    tz[i[1:], i[:-1]] = 1.0 / (dz * dz)
    tz[i[:-1], i[1:]] = 1.0 / (dz * dz)
    lam, q = torch.linalg.eigh(tz)
    w = torch.einsum("mkj,kp->jmp", y, q.to(y.dtype))                      # [j][mode][p]
    mode = torch.arange(l // 2 + 1, device=dev, dtype=f8)
    xl2 = 2.0 * (torch.cos(mode * dth) - 1.0)
    axis = torch.where(mode.remainder(2.0) == 0.0, 1.0, -1.0)
    d0 = lam[None, :]
    cp, wp = [], []
    for n in range(m_):
        d = -a[n] - c[n] + xl2[:, None] * cc[n] + d0
        if n == 0:
            d = d + (axis * a[0])[:, None]
            rhs = w[n]
        else:
            d = d - a[n] * cp[-1]
            rhs = w[n] - a[n] * wp[-1]
        cp.append((c[n] if n + 1 < m_ else 0.0) / d)
        wp.append(rhs / d)
    x = wp[-1]
    sol = [x]
    for n in range(m_ - 2, -1, -1):
        x = wp[n] - cp[n] * x
        sol.append(x)
    sol = torch.stack(sol[::-1])
    x = torch.einsum("jmp,kp->mkj", sol, q.to(sol.dtype))
    phi = torch.zeros((l, k + 2, j + 2), dtype=f8, device=dev)
    phi[:, 1:k, 1:j] = torch.fft.irfft(x, n=l, dim=0)
    phi[:, k, 1:j + 1] = bdy[:j].T
    phi[:, 1:k, j] = bdy[j:].T
    half = l // 2
    phi[:, 1:k + 1, 0] = torch.roll(phi[:, 1:k + 1, 1], half, 0)
    phi[:, 0, :j + 1] = phi[:, 1, :j + 1]
    phi[:, 1:k + 1, j + 1] = _axis_value(phi[:, 1:k + 1, 1:6], j, l, rhf)
    return phi.permute(2, 1, 0)


def exact(case, seed):
    # a step's PHI and momenta go on from what the arrays held before
    if case["kind"] == "step":
        return None
    dev = _device()
    sizes = _sizes(case)
    if dev.type == "cpu" and sum(j * k * l for j, k, l in sizes) > 3.0e7:
        return None
    return [_solve(_density(*s, 64 * seed + i, dev), *s, case["isym"]).cpu() for i, s in enumerate(sizes)]
