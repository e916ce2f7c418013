"""HLLC's energy flux at low Mach number against the flux in extended precision: element-wise constant states with
small jumps in a row of elements, where an evaluation leaves nothing but the difference of face flux and own flux.

The states are exact in binary, kappa = 1.5: density and velocities of few bits, so that the pressure, which enters
the star velocity with its jump, has no round-off of its own (eps p = 8e-15 is 1e-13 in the flux).

Bar: the star state's energy S (E* - E) is formed from the jumps, so that the flux is good to the round-off of
(E + p) u, about 110 eps = 1.3e-14, twice in the evaluation's own sums; as the difference of two energies (E = 142 at a
wave speed of 10) it is 2.4e-13.  Bar 8e-14 rms.
"""
import numpy as np
import pytest

import galaexi_gb300 as gx

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

LD = np.longdouble


def prim(U):
    U = U.astype(LD)
    u = U[..., 1] / U[..., 0]
    p = LD(0.5) * (U[..., 4] - (U[..., 1] ** 2 + U[..., 2] ** 2 + U[..., 3] ** 2) / (2 * U[..., 0]))
    return U[..., 0], u, p, U[..., 4]


def hllc_energy(UL, UR):
    """The energy flux in the x direction, left state's star region or right (subsonic)."""
    rL, uL, pL, EL = prim(UL)
    rR, uR, pR, ER = prim(UR)
    a, b = np.sqrt(rL), np.sqrt(rR)
    mean = lambda x, y: (a * x + b * y) / (a + b)  # noqa: E731
    vel = [mean(UL[..., c].astype(LD) / rL, UR[..., c].astype(LD) / rR) for c in (1, 2, 3)]
    H = mean((EL + pL) / rL, (ER + pR) / rR)
    c = np.sqrt(LD(0.5) * (H - (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2) / 2))
    SL, SR = vel[0] - c, vel[0] + c
    Ss = (pR - pL + rL * uL * (SL - uL) - rR * uR * (SR - uR)) / (rL * (SL - uL) - rR * (SR - uR))
    left = Ss >= 0
    r, u, p, E, S = (np.where(left, x, y) for x, y in ((rL, rR), (uL, uR), (pL, pR), (EL, ER), (SL, SR)))
    Es = r * (S - u) / (S - Ss) * (E / r + (Ss - u) * (Ss + p / (r * (S - u))))
    return (E + p) * u + S * (Es - E)


def test_energy_flux_of_small_jumps():
    n, rng = 64, np.random.default_rng(5)
    m = gx.Mesh(2, 2, n, 1, 1, (0.0,) * 3, (2.0 * n, 2.0, 2.0))  # unit metric terms, L_hat = 3
    rho = 1 + rng.integers(-8, 9, n) * 2.0 ** -12
    vel = np.array([0.375, 0.25, 0.125]) + rng.integers(-8, 9, (n, 3)) * 2.0 ** -12
    p = 71 + rng.integers(-8, 9, n) * 2.0 ** -12
    s = np.concatenate([rho[:, None], rho[:, None] * vel, (p / 0.5 + 0.5 * rho * (vel ** 2).sum(-1))[:, None]], -1)
    order = np.argsort(m.Elem_xGP[:, 1, 1, 1, 0])
    U = np.empty((n, 3, 3, 3, 5))
    U[order] = s[:, None, None, None, :]
    op = gx.DG(gx.config(N=2, Riemann="hllc", kappa=1.5), m)
    Ut = op.DGTimeDerivative_weakForm(0.0, torch.from_numpy(U).cuda()).cpu().numpy()[order]
    op.close()
    r, u, pe, E = prim(s)
    own = (E + pe) * u
    right = hllc_energy(s, np.roll(s, -1, 0))  # flux of the face to the right
    exact_r, exact_l = -3 * (right - own), 3 * (np.roll(right, 1) - own)
    err = np.concatenate([(Ut[:, 1, 1, 2, 4] - exact_r), (Ut[:, 1, 1, 0, 4] - exact_l)]).astype(float) / 3
    assert np.sqrt((err ** 2).mean()) <= 8e-14, np.sqrt((err ** 2).mean())
