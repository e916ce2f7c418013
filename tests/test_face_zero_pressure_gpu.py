"""The face kernel of the FP64 form where a sound speed is zero: elements of zero pressure (and temperature) beside
each other and beside ordinary ones.  The states are exact in binary, so the pressure is zero to the last bit.

Bar: the FP64 form's 1e-12 relative L2, row by row (T = 0 has a finite flux in every solver here).
"""
import numpy as np
import pytest

import galaexi_gb300 as gx
from oracle.oracle import Oracle

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def rows(cfg, m, U):
    op = gx.DG(cfg, m)
    g = op.DGTimeDerivative_weakForm(0.0, torch.from_numpy(U).cuda()).cpu().numpy()
    op.close()
    o = Oracle(cfg, m).rhs(U)
    assert np.isfinite(o).all()
    for v in range(5):
        assert np.linalg.norm(g[..., v] - o[..., v]) <= 1e-12 * np.linalg.norm(o[..., v]), v


CASES = [("lf", "none", 2), ("lf", "pi", 2), ("lf", "kg", 2), ("roeentropyfix", "none", 1), ("roeentropyfix", "pi", 1),
         ("roeentropyfix", "kg", 1), ("hllc", "none", 1)]


@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("riemann,split,cold", CASES, ids=["%s-%s" % c[:2] for c in CASES])
def test_zero_pressure(riemann, split, cold, parab):
    """`cold` neighbouring elements of zero pressure among six: with two, both states of the face between them have it
    (Roe averages are only defined when one state has a pressure)."""
    m = gx.Mesh(2, 2, 6, 1, 1, (0.0,) * 3, (1.0,) * 3)
    U = np.empty((6, 3, 3, 3, 5))
    for e in range(6):
        p, u = (0.0 if e < cold else 1.0 + e), 2.0 - 0.5 * e
        U[e] = [1.0, u, 0.5, 0.25, p / 0.4 + 0.5 * (u * u + 0.25 + 0.0625)]
    if cold < 2:  # one row of elements periodic in y and z: no face there with zero pressure on both sides
        m = gx.Mesh(2, 2, 2, 2, 2, (0.0,) * 3, (1.0,) * 3)
        U = np.concatenate([U, U[1:3]])
        for e in range(8):
            x = m.Elem_xGP[e, 1, 1, 1]
            hot = (x > 0.5).sum() > 0
            u = 1.0 + 0.5 * (x > 0.5).sum()
            U[e] = [1.0, u, 0.5, 0.25, (1.0 + e if hot else 0.0) / 0.4 + 0.5 * (u * u + 0.25 + 0.0625)]
    kw = dict(parabolic=True, mu0=1e-2) if parab else {}
    rows(gx.config(N=2, Riemann=riemann, SplitDG=split, kappa=1.4, R=1.0, **kw), m, np.ascontiguousarray(U))
