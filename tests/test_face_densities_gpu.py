"""The face kernel of the FP64 form at densities whose product is no normal number.

Bar: the FP64 form's 1e-12 relative L2, row by row.
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


# (the entropy fix takes the root of the product in the reference's formula, too)
CASES = [(r, s, u) for r, s in (("roe", "none"), ("roe", "pi"), ("roe", "kg"), ("lf", "none"))
         for u in (1e-90, 1e90)] + [("hllc", "none", 1e90)]


@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("riemann,split,units", CASES)
def test_densities_whose_product_leaves_the_range(riemann, split, parab, units):
    """Densities of 1e180 and 1e-180 (pressures of order one, T by the gas constant's unit): Roe averages."""
    rng = np.random.default_rng(3)
    m = gx.Mesh(2, 2, 4, 3, 2, (0.0,) * 3, (1.0,) * 3)
    E = m.nElems
    rho, p = rng.uniform(0.5, 2.0, E) / units ** 2, rng.uniform(0.5, 2.0, E)
    vel = rng.uniform(-1.0, 1.0, (E, 3)) * units
    U = np.concatenate([rho[:, None], rho[:, None] * vel, (p / 0.4 + 0.5 * rho * (vel ** 2).sum(-1))[:, None]], -1)
    U = np.broadcast_to(U[:, None, None, None, :], (E, 3, 3, 3, 5)) * (1 + 1e-2 * rng.standard_normal((E, 3, 3, 3, 5)))
    kw = dict(parabolic=True, mu0=1e-3 / units) if parab else {}
    rows(gx.config(N=2, Riemann=riemann, SplitDG=split, kappa=1.4, R=units ** 2, **kw), m, np.ascontiguousarray(U))
