"""The calls whose speed counts: time steps, operator evaluations and their transposes on periodic boxes.

A case is one call of a user's time loop or optimisation loop on a mesh, operator and state that the
program holds anyway:
  step      TimeStepByLSERKW2, one step in place
  cfl_step  CalcTimeStep and one step with its dt, as a loop that adapts its time step does it
  rhs       DGTimeDerivative_weakForm
  vjp       rhs_vjp, the reverse mode of one operator evaluation
`exact` states the same operator in plain torch, 64 bits, whole-array operations on
(element z, y, x, node k, j, i): nothing of this repository's is called there.
"""
import functools
import math

import numpy as np
import torch

import galaexi_gb300 as gx

KAPPA, PR = 1.4, 0.72
ETA_BR2 = 2.0


def _case(name, call, N, nx, ny, nz, flow, nodes="gauss-lobatto", split="none", riemann="lf", parabolic=True,
          lifting="br1", precision="fp64"):
    return dict(name=name, call=call, N=N, nx=nx, ny=ny, nz=nz, flow=flow, nodes=nodes, split=split, riemann=riemann,
                parabolic=parabolic, lifting=lifting, precision=precision)


def listed():
    return [
        # one evaluation on 4^3 elements at N=2, the size of the cavity regression: launches and latency
        _case("rhs_n2_gauss_4", "rhs", 2, 4, 4, 4, "tgv", nodes="gauss", riemann="roeentropyfix"),
        # the isentropic vortex of the benchmark: Euler, N=3, 8^3 elements, weak form
        _case("step_vortex_n3_8", "step", 3, 8, 8, 8, "vortex", nodes="gauss", parabolic=False),
        # the Taylor-Green regression run: 8^3 elements, N=7, a new dt at every step
        _case("cfl_step_tgv_n7_8", "cfl_step", 7, 8, 8, 8, "tgv", split="pi", riemann="roeentropyfix"),
        # an odd box at an even degree with another split form
        _case("rhs_tgv_n4_kg_7x9x11", "rhs", 4, 7, 9, 11, "tgv", split="kg"),
        # the benchmark's headline: N=7, 24^3 elements
        _case("step_tgv_n7_24", "step", 7, 24, 24, 24, "tgv", split="pi", riemann="roe"),
        # the same in the mixed form
        _case("step_tgv_n7_24_mixed", "step", 7, 24, 24, 24, "tgv", split="pi", riemann="roe", precision="mixed"),
        # curved elements on Gauss nodes with BR2, as the benchmark's second mixed case, both forms
        _case("step_curved_n5_20", "step", 5, 20, 20, 20, "curved", nodes="gauss", riemann="hllc", lifting="br2"),
        _case("step_curved_n5_20_mixed", "step", 5, 20, 20, 20, "curved", nodes="gauss", riemann="hllc", lifting="br2",
              precision="mixed"),
        # reverse mode: one stage of the benchmark's adjoint window
        _case("vjp_tgv_n5_16", "vjp", 5, 16, 16, 16, "tgv", split="pi", riemann="roe"),
    ]


def draw(rng):
    call = rng.choice(["step", "step", "step", "cfl_step", "rhs", "rhs", "vjp"])
    N = rng.randint(2, 9 if call != "vjp" else 7)
    flow = rng.choice(["tgv", "tgv", "vortex", "curved"])
    if flow == "curved":
        N = max(N, 5)  # from N=5 on the metric terms of a quadratic mapping are exact
    gauss = flow != "tgv" and rng.random() < 0.7
    split = "none" if gauss else rng.choice(["pi", "pi", "kg"] + (["none"] if call in ("rhs", "vjp") else []))
    riemann = rng.choice(["lf", "roe", "roeentropyfix"] + (["hllc"] if split == "none" else []))
    dofs = math.exp(rng.uniform(math.log(1.5e3), math.log(2.5e6)))
    side = (dofs / (N + 1) ** 3) ** (1.0 / 3.0)
    nx, ny, nz = (max(1, min(40, round(side * math.exp(rng.uniform(-0.3, 0.3))))) for _ in range(3))
    if flow == "curved":
        nx, ny, nz = max(nx, 3), max(ny, 3), max(nz, 3)
    return dict(call=call, N=N, nx=nx, ny=ny, nz=nz, flow=flow, nodes="gauss" if gauss else "gauss-lobatto", split=split,
                riemann=riemann, parabolic=flow != "vortex" and rng.random() < 0.85,
                lifting="br2" if call != "vjp" and rng.random() < 0.25 else "br1",
                precision="mixed" if call in ("step", "cfl_step") and rng.random() < 0.3 else "fp64")


def _gas(case):
    """(R, mu) of the flow; Taylor-Green: Ma 0.1, Re 1600 with T0 = 1."""
    return (71.42857, 1 / 1600.0) if case["flow"] == "tgv" else (287.058, 1e-3)


def _box(case):
    return {"tgv": (-math.pi, math.pi), "vortex": (0.0, 10.0), "curved": (0.0, 1.0)}[case["flow"]]


@functools.lru_cache(maxsize=8)
def _mesh(N, nodes, nx, ny, nz, lo, hi, deform):
    return gx.Mesh(N, 1 if nodes == "gauss" else 2, nx, ny, nz, (lo,) * 3, (hi,) * 3, deform=deform)


def _deform(case):
    return 0.05 if case["flow"] == "curved" else 0.0


def _lengths(case):
    """CFL and DFL scales of the runs that the cases are taken from (BR2 needs a smaller DFL scale)."""
    if case["flow"] == "vortex":
        return 0.9, 0.9
    return 0.8, 0.4 if case["lifting"] == "br2" else 0.8


def prepare(case, seed):
    lo, hi = _box(case)
    mesh = _mesh(case["N"], case["nodes"], case["nx"], case["ny"], case["nz"], lo, hi, _deform(case))
    R, mu = _gas(case)
    op = gx.DG(gx.config(N=case["N"], NodeType=case["nodes"], Riemann=case["riemann"], SplitDG=case["split"],
                         parabolic=case["parabolic"], mu0=mu if case["parabolic"] else 0.0, R=R, kappa=KAPPA, Pr=PR,
                         Lifting=case["lifting"], etaBR2=ETA_BR2, precision=case["precision"]), mesh)
    s = dict(case=case, op=op, U=_state(case, seed, _geometry(case)["x"]), scales=_lengths(case))
    if case["call"] in ("step", "cfl_step"):
        s["K"] = torch.zeros_like(s["U"])
    if case["call"] == "step":
        s["dt"] = _dt(case)
    if case["call"] == "vjp":
        s["Ubar"] = _cotangent(case, seed, s["U"])
    return s


def run(s):
    call, op, U = s["case"]["call"], s["op"], s["U"]
    if call == "rhs":
        return op.DGTimeDerivative_weakForm(0.0, U)
    if call == "vjp":
        return op.rhs_vjp(U, s["Ubar"])
    if call == "step":
        op.TimeStepByLSERKW2(0.0, s["dt"], U, s["K"])
        return U, s["K"]
    dt, bad = op.CalcTimeStep(U, *s["scales"])
    op.TimeStepByLSERKW2(0.0, dt, U, s["K"])
    return U, s["K"], dt, bad


def work(case):
    """Bytes: state (and RK register) in and out once per evaluation, metric terms and face geometry in.
    Operations: 1D derivative operators, two-point or pointwise fluxes, lifting, face fluxes."""
    n = case["N"] + 1
    dofs = case["nx"] * case["ny"] * case["nz"] * n ** 3
    word = 8 if case["precision"] == "fp64" else 4
    stages = 5 if case["call"] in ("step", "cfl_step") else 1
    geo = word * (10 + 30.0 / n)
    state = 160 if stages == 5 else 80
    flops = 14 + 1000.0 / n + (105 * (n - 1) if case["split"] != "none" else 30 * n) + 120
    if case["parabolic"]:
        flops += 54 * n + 115 + 500.0 / n
    if case["call"] == "vjp":
        state, flops = 120, 3 * flops
    extra = 17 * 8 if case["call"] == "cfl_step" else 0  # state and metric terms of the time step
    return {"bytes": dofs * (stages * (state + geo) + extra), "flops": dofs * stages * flops}


# ---------------------------------------------------------------------------------------------
# inputs, and the operator in plain torch
# ---------------------------------------------------------------------------------------------
def _nodes(n, kind):
    """Nodes and weights on [-1, 1], increasing."""
    P = np.polynomial.legendre
    if kind == "gauss":
        return P.leggauss(n)
    c = np.zeros(n)
    c[-1] = 1.0
    d1, d2 = P.legder(c), P.legder(c, 2)
    x = np.concatenate([[-1.0], np.sort(P.legroots(d1).real), [1.0]])
    for _ in range(4):  # Newton on P'_N
        x[1:-1] -= P.legval(x[1:-1], d1) / P.legval(x[1:-1], d2)
    x = 0.5 * (x - x[::-1])
    return x, 2.0 / (n * (n - 1) * P.legval(x, c) ** 2)


def _lagrange(x, y):
    """l_j(y_i) and l_j'(y_i) of the Lagrange basis on the points x."""
    n = len(x)
    L, D = np.ones((len(y), n)), np.zeros((len(y), n))
    for j in range(n):
        for m in range(n):
            if m == j:
                continue
            L[:, j] *= (y - x[m]) / (x[j] - x[m])
            t = np.full(len(y), 1.0 / (x[j] - x[m]))
            for q in range(n):
                if q not in (j, m):
                    t = t * (y - x[q]) / (x[j] - x[q])
            D[:, j] += t
    return L, D


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _basis(case):
    x, w = _nodes(case["N"] + 1, case["nodes"])
    D = _lagrange(x, x)[1]
    Lm, Lp = _lagrange(x, np.array([-1.0]))[0][0], _lagrange(x, np.array([1.0]))[0][0]
    Dhat = -(D.T * w[None, :]) / w[:, None]
    S = D.copy()
    S[0, 0] += 0.5 / w[0]
    S[-1, -1] -= 0.5 / w[-1]
    return {k: _dev(v) for k, v in dict(x=x, D=D, Dhat=Dhat, S=S, Lm=Lm, Lp=Lp, Lhm=Lm / w, Lhp=Lp / w).items()}


def _along(A, X, d):
    """A (rows, n) applied along the node axis of direction d (0 xi, 1 eta, 2 zeta); X (z,y,x,k,j,i,...)."""
    return torch.movedim(torch.tensordot(X, A, dims=([5 - d], [1])), -1, 5 - d)


def _geometry(case):
    """Node coordinates, contravariant metric terms, 1/J and the metric terms on the plus faces."""
    N, nel = case["N"], (case["nx"], case["ny"], case["nz"])
    lo, hi = _box(case)
    xs, _ = _nodes(N + 1, case["nodes"])
    amp = _deform(case)
    g = 3 if amp else 2
    xg = np.linspace(-1.0, 1.0, g)
    # equidistant geometry nodes of every element, displaced; shape (z, y, x, c, b, a, 3)
    c1 = [_dev(lo + (np.arange(m)[:, None] + 0.5 * (xg[None, :] + 1.0)) * ((hi - lo) / m)) for m in nel]
    shape = (nel[2], nel[1], nel[0], g, g, g)
    X = torch.stack([c1[0].view(1, 1, nel[0], 1, 1, g).expand(shape), c1[1].view(1, nel[1], 1, 1, g, 1).expand(shape),
                     c1[2].view(nel[2], 1, 1, g, 1, 1).expand(shape)], -1)
    if amp:
        X = X + amp * torch.sin(2 * math.pi * (X - lo) / (hi - lo)).prod(-1, keepdim=True)
    ends = np.array([1.0])
    L, D = (_dev(a) for a in _lagrange(xg, xs))
    L1, D1 = (_dev(a) for a in _lagrange(xg, ends))

    def at(face):
        """Tangent vectors at the solution nodes, or on the plus face of direction `face`."""
        T = []
        for d in range(3):
            Y = X
            for q in range(3):
                A = (D1 if q == d else L1) if q == face else (D if q == d else L)
                Y = _along(A, Y, q)
            T.append(Y)
        return T

    def metric(T):
        return [torch.linalg.cross(T[1], T[2]), torch.linalg.cross(T[2], T[0]), torch.linalg.cross(T[0], T[1])]

    T = at(None)
    M = metric(T)
    x = X
    for q in range(3):
        x = _along(L, x, q)
    faces = []
    for d in range(3):
        Ja = metric(at(d))[d]
        se = Ja.square().sum(-1).sqrt()
        n = Ja / se[..., None]
        ref = torch.zeros_like(n)
        ref[..., (d + 1) % 3] = 1.0
        t1 = ref - (ref * n).sum(-1, keepdim=True) * n
        t1 = t1 / t1.square().sum(-1, keepdim=True).sqrt()
        faces.append((n, t1, torch.linalg.cross(n, t1), se))
    return dict(x=x, M=M, J=(T[0] * M[0]).sum(-1), faces=faces)


def _state(case, seed, x):
    """The flow's state with a seeded part: smooth velocity modes (tgv, vortex), or noise on a uniform flow."""
    r = np.random.default_rng(seed)
    if case["flow"] == "curved":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
        vel = torch.tensor([0.3, 0.2, 0.1], dtype=torch.float64, device="cuda").expand(x.shape)
        U = _cons(torch.ones_like(x[..., 0]), vel, torch.full_like(x[..., 0], 1 / 1.4))
        U = U + 1e-3 * torch.randn(U.shape, dtype=torch.float64, device="cuda", generator=gen)
    elif case["flow"] == "vortex":
        cx, cy = 5.0 + r.uniform(-1, 1, 2)
        dx, dy = x[..., 0] - cx, x[..., 1] - cy
        du = r.uniform(0.8, 1.0) / (2 * math.pi) * torch.exp(0.5 * (1 - dx * dx - dy * dy))
        z = torch.zeros_like(du)
        T = 1 - (KAPPA - 1) / (2 * KAPPA) * du * du
        U = _cons(T ** (1 / (KAPPA - 1)), torch.stack([1 - du * dy, 1 + du * dx, z], -1), T ** (KAPPA / (KAPPA - 1)))
    else:
        X, Y, Z = x.unbind(-1)
        vel = torch.stack([torch.sin(X) * torch.cos(Y) * torch.cos(Z), -torch.cos(X) * torch.sin(Y) * torch.cos(Z),
                           torch.zeros_like(X)], -1)
        for _ in range(3):
            k, ph, amp = r.integers(1, 4, 3), r.uniform(0, 2 * math.pi), _dev(0.03 * r.standard_normal(3))
            vel = vel + torch.sin(k[0] * X + k[1] * Y + k[2] * Z + ph)[..., None] * amp
        p = 100.0 / KAPPA + (torch.cos(2 * X) * torch.cos(2 * Z) + 2 * torch.cos(2 * Y) + 2 * torch.cos(2 * X)
                             + torch.cos(2 * Y) * torch.cos(2 * Z)) / 16.0
        U = _cons(torch.ones_like(X), vel, p)
    return U.reshape(-1, *U.shape[3:]).contiguous()


def _cons(rho, vel, p):
    return torch.cat([rho[..., None], rho[..., None] * vel,
                      (p / (KAPPA - 1) + 0.5 * rho * vel.square().sum(-1))[..., None]], -1)


def _cotangent(case, seed, U):
    """What an optimisation of the kinetic energy sends back: its derivative, plus seeded noise."""
    gen = torch.Generator(device="cuda").manual_seed((int(seed) + 17) % (1 << 62))
    vel = U[..., 1:4] / U[..., :1]
    g = torch.cat([-0.5 * vel.square().sum(-1, keepdim=True), vel, torch.zeros_like(U[..., :1])], -1)
    return g + 1e-3 * torch.randn(U.shape, dtype=torch.float64, device="cuda", generator=gen)


def _alphas(case):
    """CFL and DFL limits of the five-stage scheme for N = 1..9 (Gauss, Gauss-Lobatto)."""
    cfl = {"gauss": [2.0351, 1.7595, 1.5401, 1.3702, 1.2375, 1.1318, 1.0440, 0.9709, 0.9079],
           "gauss-lobatto": [4.7497, 3.4144, 2.8451, 2.4739, 2.2027, 1.9912, 1.8225, 1.6830, 1.5682]}
    dfl = {"gauss": [1.12, 0.76, 0.55, 0.41, 0.32, 0.25, 0.20, 0.17, 0.14],
           "gauss-lobatto": [4.50, 1.95, 1.18, 0.79, 0.56, 0.42, 0.32, 0.25, 0.20]}
    i, m = case["N"] - 1, 2.0 * case["N"] + 1
    return cfl[case["nodes"]][i] / m, dfl[case["nodes"]][i] * 1.853 / m ** 2


def _dt(case):
    """A dt below the limits for the flow's largest velocities, fixed over the run."""
    lo, hi = _box(case)
    h = (hi - lo) / max(case["nx"], case["ny"], case["nz"])
    c = {"tgv": 10.3, "vortex": 1.2, "curved": 1.05}[case["flow"]]
    v = {"tgv": 2.5, "vortex": 2.3, "curved": 0.7}[case["flow"]]
    (s, d), (ac, ad) = _lengths(case), _alphas(case)
    dt = s * ac * h / (3 * c + v) * (0.6 if case["flow"] == "curved" else 1.0)
    if case["parabolic"]:
        dt = min(dt, d * ad * h * h / (3 * _gas(case)[1] * KAPPA / PR) * (0.4 if case["flow"] == "curved" else 0.9))
    return dt


def _prim(U, R):
    vel = U[..., 1:4] / U[..., :1]
    p = (KAPPA - 1) * (U[..., 4] - 0.5 * (U[..., 1:4] * vel).sum(-1))
    return vel, p, p / (U[..., 0] * R)


def _stress(G, vel, mu, lam):
    """Rows d of -(tau_d, tau_d . v + lam dT/dx_d): (..., 3, 4) from G (..., 3, 4), d/dx_d of (u, v, w, T)."""
    g = G[..., :3]
    div = g[..., 0, 0] + g[..., 1, 1] + g[..., 2, 2]
    tau = mu * (g + g.transpose(-1, -2)) - (2.0 / 3.0) * mu * div[..., None, None] * torch.eye(3, dtype=g.dtype, device=g.device)
    return -torch.cat([tau, ((tau * vel[..., None, :]).sum(-1) + lam * G[..., 3])[..., None]], -1)


def _riemann(case, UL, UR, n, t1, t2, R):
    """Flux through faces with unit normals n (element on the left of n: UL)."""
    def ext(U):
        vel, p, _ = _prim(U, R)
        return U[..., 0], (vel * n).sum(-1), (vel * t1).sum(-1), (vel * t2).sum(-1), U[..., 4], p
    (rL, uL, vL, wL, EL, pL), (rR, uR, vR, wR, ER, pR) = ext(UL), ext(UR)
    stack = lambda *a: torch.stack(a, -1)  # noqa: E731
    FL = stack(rL * uL, rL * uL * uL + pL, rL * uL * vL, rL * uL * wL, (EL + pL) * uL)
    FR = stack(rR * uR, rR * uR * uR + pR, rR * uR * vR, rR * uR * wR, (ER + pR) * uR)
    HL, HR = (EL + pL) / rL, (ER + pR) / rR
    if case["split"] == "none":
        F = 0.5 * (FL + FR)
    else:
        q = 0.125 * (rL + rR) * (uL + uR)
        e = q * (HL + HR) if case["split"] == "pi" else q * (EL / rL + ER / rR) + 0.25 * (pL + pR) * (uL + uR)
        F = stack(2 * q, q * (uL + uR) + 0.5 * (pL + pR), q * (vL + vR), q * (wL + wR), e)
    cL, cR = (KAPPA * pL / rL).sqrt(), (KAPPA * pR / rR).sqrt()
    kind = case["riemann"]
    if kind == "lf":
        lam = torch.maximum(uL.abs(), uR.abs()) + torch.maximum(cL, cR)
        dU = stack(rR - rL, rR * uR - rL * uL, rR * vR - rL * vL, rR * wR - rL * wL, ER - EL)
        F = F - 0.5 * lam[..., None] * dU
    else:
        a, b = rL.sqrt(), rR.sqrt()
        u, v, w, H = ((b * y + a * x) / (a + b) for x, y in ((uL, uR), (vL, vR), (wL, wR), (HL, HR)))
        q2 = u * u + v * v + w * w
        c = ((KAPPA - 1) * (H - 0.5 * q2)).sqrt()
        if kind == "hllc":
            Sl, Sr = u - c, u + c
            ml, mr = rL * (Sl - uL), rR * (Sr - uR)
            Ss = (pR - pL + ml * uL - mr * uR) / (ml - mr)

            def star(r, un, vt, wt, E, p, S, m, F0):
                f = m / (S - Ss)
                Us = stack(f, f * Ss, f * vt, f * wt, f * (E / r + (Ss - un) * (Ss + p / m)))
                return F0 + S[..., None] * (Us - stack(r, r * un, r * vt, r * wt, E))
            F = torch.where((Ss >= 0)[..., None], star(rL, uL, vL, wL, EL, pL, Sl, ml, FL),
                            star(rR, uR, vR, wR, ER, pR, Sr, mr, FR))
            F = torch.where((Sl >= 0)[..., None], FL, torch.where((Sr <= 0)[..., None], FR, F))
        else:
            d = a * b
            dr, du, dv, dw, dp = rR - rL, uR - uL, vR - vL, wR - wL, pR - pL
            lam = [u - c, u, u, u, u + c]
            if kind == "roeentropyfix":
                for i, (l, r) in enumerate(zip((uL - cL, uL, uL, uL, uL + cL), (uR - cR, uR, uR, uR, uR + cR))):
                    da = torch.clamp(torch.maximum(lam[i] - l, r - lam[i]), min=0.0)
                    s = torch.where(da > 0, da, torch.ones_like(da))
                    lam[i] = torch.where(lam[i].abs() < da, 0.5 * (lam[i] * lam[i] / s + da), lam[i].abs())
            else:
                lam = [x.abs() for x in lam]
                # Roe on conserved jumps: the same wave strengths from (r, m, E) differences
                g = [dr, rR * uR - rL * uL, rR * vR - rL * vL, rR * wR - rL * wL, ER - EL]
                A3, A4 = g[2] - v * g[0], g[3] - w * g[0]
                A2 = (KAPPA - 1) / (c * c) * (g[0] * (H - u * u) - (g[4] - A3 * v - A4 * w) + u * g[1])
                A1 = 0.5 / c * (g[0] * (u + c) - g[1] - c * A2)
                A5 = g[0] - A1 - A2
            if kind == "roeentropyfix":
                t = 0.5 / (c * c)
                A1, A2, A3, A4, A5 = t * (dp - d * c * du), dr - 2 * t * dp, d * dv, d * dw, t * (dp + d * c * du)
            w1, w2, w3, w4, w5 = A1 * lam[0], A2 * lam[1], A3 * lam[2], A4 * lam[3], A5 * lam[4]
            F = F - 0.5 * stack(w1 + w2 + w5, w1 * (u - c) + w2 * u + w5 * (u + c), (w1 + w2 + w5) * v + w3,
                                (w1 + w2 + w5) * w + w4,
                                w1 * (H - u * c) + w2 * 0.5 * q2 + w3 * v + w4 * w + w5 * (H + u * c))
    m = F[..., 1:2] * n + F[..., 2:3] * t1 + F[..., 3:4] * t2
    return torch.cat([F[..., :1], m, F[..., 4:]], -1)


def _pair_volume(case, b, U, M, R):
    """Split form: sum over the nodes of each line of DVolSurf times the two-point flux."""
    vel, p, _ = _prim(U, R)
    rho, E = U[..., 0], U[..., 4]
    aux = (E + p) / rho if case["split"] == "pi" else E / rho
    out = torch.zeros_like(U)
    for d in range(3):
        ax = 5 - d
        pair = lambda q: q.unsqueeze(ax + 1) + q.unsqueeze(ax)  # noqa: E731  (node, partner) on axes ax, ax+1
        rs, us, ps, xs, Ms = pair(rho), pair(vel), pair(p), pair(aux), pair(M[d])
        Vs = (Ms * us).sum(-1)
        q = 0.125 * rs * Vs
        e = q * xs + (0.25 * ps * Vs if case["split"] == "kg" else 0.0)
        F = torch.cat([2 * q[..., None], q[..., None] * us + 0.5 * ps[..., None] * Ms, e[..., None]], -1)
        n = b["S"].shape[0]
        view = [1] * F.dim()
        view[ax] = view[ax + 1] = n
        S = b["S"] - torch.diag(torch.diag(b["S"]))
        out = out + (S.view(view) * F).sum(ax + 1)
    return out


def _rhs(case, b, geo, U, mu):
    """Ut of U (z,y,x,k,j,i,5); mu a number or a tensor that gradients are taken for."""
    R = _gas(case)[0]
    lam = mu * R * KAPPA / ((KAPPA - 1) * PR)
    M, sJ, faces = geo["M"], 1.0 / geo["J"], geo["faces"]
    plus = lambda X, d: _along(b["Lp"][None], X, d)  # noqa: E731
    minus = lambda X, d: _along(b["Lm"][None], X, d)  # noqa: E731
    right = lambda X, d: torch.roll(X, -1, 2 - d)  # noqa: E731  (the next element's values)
    left = lambda X, d: torch.roll(X, 1, 2 - d)  # noqa: E731

    def lift(X, d, Fp, Fm):
        """L_hat times the plus face's and minus face's values, on the nodes of the lines of direction d."""
        return _along(b["Lhp"][:, None], Fp, d) + _along(b["Lhm"][:, None], Fm, d)

    vel, p, T = _prim(U, R)
    UL = [plus(U, d) for d in range(3)]
    UR = [right(minus(U, d), d) for d in range(3)]
    if case["parabolic"]:
        def lifted(X):
            v, _, t = _prim(X, R)
            return torch.cat([v, t[..., None]], -1)
        Q = torch.cat([vel, T[..., None]], -1)
        G = sum(M[d][..., :, None] * _along(b["D"], Q, d)[..., None, :] for d in range(3))
        # 0.5 SurfElem (slave - master) n on the plus faces; the same on the slave's minus face
        J = [0.5 * faces[d][3][..., None, None] * faces[d][0][..., :, None] * (lifted(UR[d]) - lifted(UL[d]))[..., None, :]
             for d in range(3)]
        GV = G * sJ[..., None, None]
        own = [(_along(b["Lhp"][:, None], J[d], d), _along(b["Lhm"][:, None], left(J[d], d), d)) for d in range(3)]
        G = (G + sum(a + c for a, c in own)) * sJ[..., None, None]
        if case["lifting"] == "br2":
            GL = [plus(GV + ETA_BR2 * own[d][0] * sJ[..., None, None], d) for d in range(3)]
            GR = [right(minus(GV + ETA_BR2 * own[d][1] * sJ[..., None, None], d), d) for d in range(3)]
        else:
            GL = [plus(G, d) for d in range(3)]
            GR = [right(minus(G, d), d) for d in range(3)]
    out = torch.zeros_like(U)
    if case["split"] != "none":
        out = out + _pair_volume(case, b, U, M, R)
    else:
        F = torch.cat([U[..., None, 1:4].transpose(-1, -2), U[..., 1:4, None] * vel[..., None, :]
                       + p[..., None, None] * torch.eye(3, dtype=U.dtype, device=U.device),
                       ((U[..., 4] + p)[..., None] * vel)[..., None]], -1)
        for d in range(3):
            out = out + _along(b["Dhat"], (M[d][..., :, None] * F).sum(-2), d)
    if case["parabolic"]:
        V = _stress(G, vel, mu, lam)
        for d in range(3):
            f = _along(b["Dhat"], (M[d][..., :, None] * V).sum(-2), d)
            out = out + torch.cat([torch.zeros_like(f[..., :1]), f], -1)
    for d in range(3):
        n, t1, t2, se = faces[d]
        F = _riemann(case, UL[d], UR[d], n, t1, t2, R)
        if case["parabolic"]:
            f = 0.5 * sum((n[..., :, None] * _stress(g, _prim(u, R)[0], mu, lam)).sum(-2)
                          for g, u in ((GL[d], UL[d]), (GR[d], UR[d])))
            F = F + torch.cat([torch.zeros_like(f[..., :1]), f], -1)
        F = F * se[..., None]
        out = out + lift(U, d, F, -left(F, d))
    return -out * sJ[..., None]


def _cfl_dt(case, geo, U):
    cfl, dfl = (s * a for s, a in zip(_lengths(case), _alphas(case)))
    vel, p, _ = _prim(U, _gas(case)[0])
    c, sJ = (KAPPA * p / U[..., 0]).sqrt(), 1.0 / geo["J"]
    a, v = 0.0, 0.0
    for d in range(3):
        m = geo["M"][d] * sJ[..., None]
        ld = (m * vel).sum(-1).abs() + c * m.square().sum(-1).sqrt()
        a = a + ld.amax((3, 4, 5))
        v = v + (max(4 / 3, KAPPA / PR) * _gas(case)[1] / U[..., 0] * m.square().sum(-1)).amax((3, 4, 5))
    dt = float((cfl * 2.0 / a).min())
    return min(dt, float((dfl * 4.0 / v).min())) if case["parabolic"] else dt


_A = (0.0, 567301805773.0 / 1357537059087.0, 2404267990393.0 / 2016746695238.0, 3550918686646.0 / 2091501179385.0,
      1275806237668.0 / 842570457699.0)
_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, 1720146321549.0 / 2090206949498.0,
      3134564353537.0 / 4481467310338.0, 2277821191437.0 / 14882151754819.0)


def exact(case, seed):
    b, geo = _basis(case), _geometry(case)
    U = _state(case, seed, geo["x"])
    shape = U.shape
    cells = (case["nz"], case["ny"], case["nx"])
    mu = _gas(case)[1] if case["parabolic"] else 0.0
    if case["call"] == "vjp":
        X = U.view(*cells, *shape[1:]).clone().requires_grad_()
        m = torch.tensor(mu, dtype=torch.float64, device="cuda", requires_grad=True)
        Ut = _rhs(case, b, geo, X, m)
        g = torch.autograd.grad(Ut, [X, m], _cotangent(case, seed, U).view(X.shape), allow_unused=True)
        return g[0].reshape(shape), float(g[1]) if g[1] is not None else 0.0
    with torch.no_grad():
        X = U.view(*cells, *shape[1:])
        if case["call"] == "rhs":
            return _rhs(case, b, geo, X, mu).reshape(shape)
        dt = _cfl_dt(case, geo, X) if case["call"] == "cfl_step" else _dt(case)
        K = torch.zeros_like(X)
        for s in range(5):
            K = _rhs(case, b, geo, X, mu) - _A[s] * K
            X = X + _B[s] * dt * K
        out = (X.reshape(shape), K.reshape(shape))
        return out + (dt, 0) if case["call"] == "cfl_step" else out
