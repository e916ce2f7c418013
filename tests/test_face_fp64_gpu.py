"""The face kernel of the FP64 form (csrc/dg_face_fx.cuh) against the oracle where its branches lie: element-wise
constant random states with jumps up to a factor of four, sub- and supersonic in every direction (the
one-sided fluxes of HLLC, the entropy fix), units far from one (the exponent handling of the reciprocals and
square roots), and values beyond the range of the FP32 approximations.

Bar: the FP64 form's 1e-12 relative L2 per evaluation.
"""
import zlib

import numpy as np
import pytest

import galaexi_gb300 as gx
from oracle.oracle import Oracle

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

KAPPA = 1.4


def piecewise_state(m, seed, units):
    rng = np.random.default_rng(zlib.crc32(seed.encode()))
    E = m.nElems
    rho, p = rng.uniform(0.5, 2.0, E), rng.uniform(0.5, 2.0, E)
    vel = rng.uniform(-4.0, 4.0, (E, 3)) * (rng.random((E, 1)) < 0.7)
    D, V = units ** -2, units
    rho, vel, p = rho * D, vel * V, p * D * V * V
    U = np.concatenate([rho[:, None], rho[:, None] * vel, (p / (KAPPA - 1) + 0.5 * rho * (vel ** 2).sum(-1))[:, None]], -1)
    n = m.N + 1
    U = np.broadcast_to(U[:, None, None, None, :], (E, n, n, n, 5)).copy()
    return U * (1 + 1e-2 * rng.standard_normal(U.shape))


CASES = [(r, s) for r in ("lf", "roe", "roeentropyfix") for s in ("none", "pi", "kg")] + [("hllc", "none")]


@pytest.mark.parametrize("units", [1.0, 1e-30, 1e40])
@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("riemann,split", CASES, ids=["%s-%s" % c for c in CASES])
def test_strong_jumps(riemann, split, parab, units):
    N = 2
    m = gx.Mesh(N, 2, 4, 3, 3, (0.0,) * 3, (1.0,) * 3, deform=0.04)
    kw = dict(parabolic=True, mu0=1e-3 / units) if parab else {}
    # (R scales so that T = p / (rho R) stays of order one)
    cfg = gx.config(N=N, Riemann=riemann, SplitDG=split, R=units ** 2, kappa=KAPPA, **kw)
    U = piecewise_state(m, riemann + split, units)
    op = gx.DG(cfg, m)
    g = op.DGTimeDerivative_weakForm(0.0, torch.from_numpy(U).cuda()).cpu().numpy()
    op.close()
    o = Oracle(cfg, m).rhs(U)
    for v in range(5):  # the rows differ by powers of the units
        a, b = g[..., v], o[..., v]
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b), (v, np.linalg.norm(a - b) / np.linalg.norm(b))
