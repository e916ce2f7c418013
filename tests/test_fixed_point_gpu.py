"""The fixed-point kernels of the FP64 form (csrc/dg_fx.cuh) against the oracle where their scales are
chosen or given up: units far from one, fluid at rest, viscous and pressure dominated flow, flat elements,
and elements that leave the fixed-point path (contrasts beyond 2^8 in density or pressure, values outside
2^+-150, NaN).

Bar: the FP64 form's 1e-12 relative L2 per evaluation (5e-12 where the flux differences of the case cancel to
less than a thousandth of the fluxes, as for the fluid at rest).
"""
import math
import zlib

import numpy as np
import pytest

import galaexi_gb300 as gx
from oracle.oracle import Oracle

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

R = 71.42857


def gpu_rhs(cfg, m, U):
    op = gx.DG(cfg, m)
    Ut = op.DGTimeDerivative_weakForm(0.0, torch.from_numpy(U.copy()).cuda()).cpu().numpy()
    op.close()
    return Ut


def state(m, seed, mach=0.3, noise=1e-2):
    rng = np.random.default_rng(zlib.crc32(seed.encode()))
    U = gx.tgv_state(m, mach=mach, R=R)
    return U + noise * rng.standard_normal(U.shape) * np.abs(U).mean(axis=(0, 1, 2, 3))


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


FORMS = [("pi", dict(SplitDG="pi", Riemann="roe")), ("kg", dict(SplitDG="kg", Riemann="lf")),
         ("weak", dict(Riemann="roe")), ("gauss", dict(NodeType="gauss", Riemann="lf")),
         ("gauss_br2", dict(NodeType="gauss", Riemann="lf", Lifting="br2")),
         ("pi_br2", dict(SplitDG="pi", Riemann="roe", Lifting="br2"))]


@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("form,kw", FORMS, ids=[f[0] for f in FORMS])
@pytest.mark.parametrize("N,units", [(2, 1e-4), (3, 1e5), (5, 1e-6), (6, 1e3), (7, 1e-3), (8, 1e2), (9, 1e-2)])
def test_units(N, units, form, kw, parab):
    """Lengths in `units`, velocities in sqrt(units), density in 1/units: every scale moves by its own power."""
    L, V, D = units, math.sqrt(units), 1.0 / units
    nt = 1 if "NodeType" in kw else 2
    m = gx.Mesh(N, nt, 2, 1, 2, (-math.pi * L,) * 3, (math.pi * L,) * 3, deform=0.0)
    m1 = gx.Mesh(N, nt, 2, 1, 2, (-math.pi,) * 3, (math.pi,) * 3)
    U = state(m1, "units%d%s" % (N, form)) * np.array([D, D * V, D * V, D * V, D * V * V])
    k = dict(kw, parabolic=True, mu0=2e-3 * D * V * L) if parab else kw
    cfg = gx.config(N=N, R=R, **k)
    assert rel(gpu_rhs(cfg, m, U), Oracle(cfg, m).rhs(U)) <= 1e-12


@pytest.mark.parametrize("what", ["mach0.01", "viscous", "flat", "supersonic"])
@pytest.mark.parametrize("nodes", ["split", "weak", "gauss"])
@pytest.mark.parametrize("N", [4, 7])
def test_dominant_terms(N, nodes, what):
    lo, hi = (-math.pi,) * 3, (math.pi,) * 3
    if what == "flat":
        lo, hi = (-math.pi, -1e-3, -math.pi), (math.pi, 1e-3, math.pi)
    m = gx.Mesh(N, 1 if nodes == "gauss" else 2, 2, 2, 1, lo, hi)
    mach = {"mach0.01": 0.01, "supersonic": 3.0}.get(what, 0.3)
    noise = 1e-4 if what == "supersonic" else 1e-2
    U = state(m, what, mach=1.0 if what == "supersonic" else mach, noise=noise)
    if what == "supersonic":
        U[..., 4] += 2.0 * np.abs(U[..., 1]) ** 2 / U[..., 0]
        U[..., 4] += 6.0 * U[..., 1] + 18.0 * U[..., 0]  # a uniform velocity on top, exactly
        U[..., 1] += 6.0 * U[..., 0]
    cfg = gx.config(N=N, R=R, SplitDG="pi" if nodes == "split" else "none", Riemann="roe", parabolic=True,
                    NodeType="gauss" if nodes == "gauss" else "gauss-lobatto", mu0=1.0 if what == "viscous" else 2e-3)
    assert rel(gpu_rhs(cfg, m, U), Oracle(cfg, m).rhs(U)) <= 1e-12


def test_at_rest():
    """Zero velocities and velocity gradients: the groups without a magnitude."""
    m = gx.Mesh(5, 2, 2, 2, 2, (-math.pi,) * 3, (math.pi,) * 3)
    U = gx.fill_ini(m, 1, [1.0, 0.0, 0.0, 0.0, 1 / 1.4])
    U[..., 0] *= 1 + 1e-2 * np.sin(m.Elem_xGP[..., 0])
    U[..., 4] *= 1 + 1e-1 * np.sin(m.Elem_xGP[..., 1])
    cfg = gx.config(N=5, R=R, SplitDG="pi", Riemann="roe", parabolic=True, mu0=2e-3)
    assert rel(gpu_rhs(cfg, m, U), Oracle(cfg, m).rhs(U)) <= 5e-12


@pytest.mark.parametrize("form,kw", FORMS, ids=[f[0] for f in FORMS])
@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("what", ["density", "pressure", "tiny"])
@pytest.mark.parametrize("N", [3, 6, 7])
def test_elements_outside_the_scales(N, what, parab, form, kw):
    """One element with a contrast beyond one scale (or magnitudes below 2^-150) among ordinary ones."""
    m = gx.Mesh(N, 1 if "NodeType" in kw else 2, 2, 2, 1, (-math.pi,) * 3, (math.pi,) * 3)
    U = state(m, "outside" + what)
    x = m.Elem_xGP[1, ..., 0:1] * np.array([1.0])
    s = (x - x.min()) / (x.max() - x.min())
    if what == "density":
        U[1] *= 2000.0 ** s  # rho, m, E together: velocities stay, the pressure follows
    elif what == "pressure":
        U[1, ..., 4:] *= 2000.0 ** s
    else:
        U *= 1e-50
    k = dict(kw, parabolic=True, mu0=2e-3 * (1e-50 if what == "tiny" else 1.0)) if parab else kw
    cfg = gx.config(N=N, R=R, **k)
    assert rel(gpu_rhs(cfg, m, U), Oracle(cfg, m).rhs(U)) <= 1e-12


@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_non_finite_values_stay_on_their_lines(bad):
    N = 5
    m = gx.Mesh(N, 2, 2, 2, 2, (-math.pi,) * 3, (math.pi,) * 3)
    U = state(m, "nan")
    U[3, 2, 3, 1, 4] = bad  # the energy of an inner node
    cfg = gx.config(N=N, R=R, SplitDG="pi", Riemann="roe")
    g = gpu_rhs(cfg, m, U)
    lines = np.zeros(U.shape[:4], dtype=bool)
    lines[3, 2, 3, :] = lines[3, 2, :, 1] = lines[3, :, 3, 1] = True
    assert np.array_equal(~np.isfinite(g).all(axis=-1), lines)
    o = Oracle(cfg, m).rhs(U)
    assert rel(g[~lines], o[~lines]) <= 1e-12
