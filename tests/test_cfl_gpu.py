"""k_cfl: the maxima over an element's nodes (whole and partial warps, one to 32 warps) and nodes without a number.

Bar: the time step is a maximum of FP64 expressions of a dozen operations each, 1e-13 relative.
"""
import math

import numpy as np
import pytest

import galaexi_gb300 as gx
from oracle.oracle import Oracle

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

R = 71.42857


def timestep(cfg, m, U):
    op = gx.DG(cfg, m)
    dt, bad = op.CalcTimeStep(torch.from_numpy(U).cuda(), 0.8, 0.4)
    op.close()
    return dt, bad


@pytest.mark.parametrize("parab", [False, True], ids=["euler", "ns"])
@pytest.mark.parametrize("N", [1, 2, 3, 6, 9])
def test_timestep(N, parab):
    m = gx.Mesh(N, 2, 2, 3, 1, (-math.pi,) * 3, (math.pi,) * 3)
    rng = np.random.default_rng(N)
    U = gx.tgv_state(m, mach=0.3, R=R)
    U = U + 1e-2 * rng.standard_normal(U.shape) * np.abs(U).mean(axis=(0, 1, 2, 3))
    cfg = gx.config(N=N, R=R, parabolic=parab, mu0=0.1 if parab else 0.0)
    dt, bad = timestep(cfg, m, U)
    ref, _ = Oracle(cfg, m).calc_timestep(U, 0.8, 0.4)
    assert bad == 0 and abs(dt - ref) <= 1e-13 * ref

    # a node without a number counts as bad and leaves the maxima to the others
    quiet = U.copy()
    quiet[1, 0, 1, 0] = (1.0, 0.0, 0.0, 0.0, 1e-6)
    dt_q, _ = timestep(cfg, m, quiet)
    quiet[1, 0, 1, 0, 4] = math.nan
    dt_n, bad = timestep(cfg, m, quiet)
    assert bad != 0 and dt_n == dt_q
