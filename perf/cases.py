"""The workloads whose speed is followed: what a user of the framework has it
do, through its public entry points, over the range of mesh sizes, orders,
element shapes, boundary conditions, precisions and directions it serves.

A case is a dict of plain values:
  kind    "step"      set_state_device, step (RK steps with their printed norms), get_state_device
          "host"      step_host: steps of a state in page-locked host memory
          "residual"  residual_device: R and f = -Minv R of a nodal state
          "vjp"       autograd.residual, forward and backward
          "adjoint"   autograd.integrate, forward and backward, with the parameter gradients
  nx ny nz p q, shape ("box", "shear": affine parallelepipeds, "sine": curved,
  "bump": the bump channel), flow (the initial state and its constants),
  sides (the boundary conditions), precision, scheme, steps, slots
  (checkpoints of the adjoint), pr (Prandtl number, 0: no heat flux)

`exact` is the same discretisation in dense torch float64, written from the
equations alone; gradients of it come from torch's own differentiation.
"""
import math

import numpy as np
import torch

import dgpr_b200 as dg
from dgpr_b200 import autograd as ag

TWO_PI = 2.0 * math.pi
PER, FREE, WALL, INFLOW, OUTFLOW, NOSLIP, ISO = -2, -3, -4, -5, -6, -7, -8
SIDES = {  # -x +x -y +y -z +z
    "periodic": [PER] * 6,
    "freestream": [FREE, FREE, FREE, FREE, PER, PER],
    "noslip": [PER, PER, NOSLIP, NOSLIP, PER, PER],
    "isothermal": [PER, PER, ISO, ISO, PER, PER],
    "throughflow": [INFLOW, OUTFLOW, WALL, WALL, PER, PER],
}


def _case(name, kind, n, p, flow, *, q=1, shape="box", sides="periodic", precision="fp64", scheme="RK4", steps=1,
          slots=0, pr=0.0):
    c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "p": p, "q": q, "shape": shape, "flow": flow,
         "sides": sides, "precision": precision, "scheme": scheme, "steps": steps, "slots": slots, "pr": pr}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the isentropic vortex at its own size: a small Euler run, where launches and latency count
        _case("vortex_8_p2", "step", (8, 8, 8), 2, "vortex", steps=10),
        # the benchmark's workload, the Taylor-Green vortex, in both precisions
        _case("tgv_32_p3", "step", (32, 32, 32), 3, "tgv", steps=5),
        _case("tgv_32_p3_mixed", "step", (32, 32, 32), 3, "tgv", precision="mixed", steps=5),
        # the largest: the same flow at order 4 on 48^3
        _case("tgv_48_p4_mixed", "step", (48, 48, 48), 4, "tgv", precision="mixed", steps=2),
        # a state that lives in host memory, one step a call
        _case("tgv_32_p3_host", "host", (32, 32, 32), 3, "tgv", steps=1),
        # the wall-bounded channel on curved elements with heat flux, full size, TVD-RK3
        _case("channel_64x32x32_p3", "step", (64, 32, 32), 3, "channel", q=2, shape="sine", sides="isothermal",
              scheme="tvdRK3", steps=2, pr=0.71),
        # a smaller one with the reference's walls, mixed precision and an odd element count
        _case("channel_25x17x13_p3_mixed", "step", (25, 17, 13), 3, "channel", q=2, shape="sine", sides="noslip",
              precision="mixed", scheme="tvdRK3", steps=4),
        # the bump channel with in- and outflow, the driver's stock geometry
        _case("bump_16_p3", "step", (16, 16, 16), 3, "stream", q=2, shape="bump", sides="throughflow", steps=5),
        # a high order on an odd-sided box with heat flux, mixed precision
        _case("box_11x9x10_p5_mixed", "step", (11, 9, 10), 5, "fourier", precision="mixed", steps=3, pr=0.71),
        # one residual, as a caller with a time scheme of their own asks for it
        _case("residual_13x11x9_p2", "residual", (13, 11, 9), 2, "stream", shape="shear", sides="freestream"),
        # a residual inside a torch graph, forward and backward
        _case("vjp_12_p4", "vjp", (12, 12, 12), 4, "fourier"),
        # gradients through a run with few checkpoints: the adjoint configuration's mesh and flow
        _case("adjoint_16_p3", "adjoint", (16, 16, 16), 3, "fourier", steps=10, slots=4),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["host", "residual", "vjp", "adjoint", "adjoint"])
    p = rng.choice([1, 2, 2, 3, 3, 3, 3, 4, 4, 5, 6])
    # values of a state, and steps so that a pass stays below the largest listed one's work
    values = math.exp(rng.uniform(math.log(2e4), math.log(6e6)))
    side = (values / (5 * (p + 1) ** 3)) ** (1.0 / 3.0)
    n = [max(2, round(side * math.exp(rng.uniform(-0.5, 0.5)))) for _ in range(3)]
    shape, q = rng.choice([("box", 1), ("box", 1), ("box", 2), ("shear", 1), ("sine", 2), ("bump", 2)])
    if shape == "sine":
        sides = rng.choice(["periodic", "noslip", "isothermal"])
    elif shape == "bump":
        sides = rng.choice(["throughflow", "noslip"])
    elif shape == "shear":
        sides = rng.choice(["periodic", "freestream"])
    else:
        sides = rng.choice(["periodic", "periodic", "freestream", "noslip", "isothermal"])
    flow = ("stream" if sides in ("freestream", "throughflow") else "channel" if sides != "periodic" else
            rng.choice(["tgv", "fourier"] if shape in ("sine", "shear") else ["tgv", "fourier", "vortex"]))
    steps = rng.randint(1, 6) if kind in ("step", "host", "adjoint") else 1
    # (the adjoint and the residual's product run in FP64 on a handle of either precision)
    precision = rng.choice(["fp64", "fp64", "mixed"]) if kind in ("step", "host", "adjoint") else "fp64"
    return _case(None, kind, n, p, flow, q=q, shape=shape, sides=sides, precision=precision,
                 scheme=rng.choice(["RK4", "RK4", "tvdRK3"]), steps=steps,
                 slots=rng.randint(1, steps) if kind == "adjoint" else 0,
                 pr=rng.choice([0.0, 0.0, 0.71]) if flow != "vortex" else 0.0)


# ------------------------------------------------------------------ the inputs

def _constants(c):
    """Extents and the reference state (gamma 1.4, R 287, eta 6) of a flow."""
    flow = c["flow"]
    if flow == "vortex":
        return dict(l=(10.0, 10.0, 10.0), mu=0.0, c=math.sqrt(1.4), u=1.0, v=1.0, w=0.0, src=0.0)
    if flow == "tgv":
        return dict(l=(TWO_PI,) * 3, mu=1.0 / 1600.0, c=10.0, u=0.0, v=0.0, w=0.0, src=0.0)
    if flow == "fourier":
        return dict(l=(TWO_PI,) * 3, mu=0.002, c=10.0 / 3.0, u=1.0, v=0.0, w=0.0, src=0.0)
    if flow == "channel":
        nu = 2.0 / 5600.0
        return dict(l=(2 * TWO_PI, 2.0, TWO_PI), mu=nu, c=5.0, u=0.0, v=0.0, w=0.0, src=(180.0 * nu) ** 2)
    return dict(l=(2.0, 1.0, 1.0), mu=1e-3, c=1.0, u=0.1, v=0.0, w=0.0, src=0.0)  # "stream": the driver's defaults


def _nodes(c):
    """Element nodes [E][z][y][x][3], equispaced per element."""
    nx, ny, nz, q = c["nx"], c["ny"], c["nz"], c["q"]
    lx, ly, lz = _constants(c)["l"]
    a = np.arange(q + 1) / q
    x = (np.arange(nx)[:, None] + a) * (lx / nx)
    y = (np.arange(ny)[:, None] + a) * (ly / ny)
    z = (np.arange(nz)[:, None] + a) * (lz / nz)
    X = np.empty((nz, ny, nx, q + 1, q + 1, q + 1, 3))
    X[..., 0] = x[None, None, :, None, None, :]
    X[..., 1] = y[None, :, None, None, :, None]
    X[..., 2] = z[:, None, None, :, None, None]
    if c["shape"] == "shear":
        X[..., 0] += 0.3 * X[..., 1]
    elif c["shape"] == "sine":
        d = 0.05 * ly / 2 * np.sin(TWO_PI * X[..., 0] / lx) * np.sin(TWO_PI * X[..., 2] / lz)
        if c["sides"] != "periodic":
            d = d * (1.0 - (2.0 * X[..., 1] / ly - 1.0) ** 2)
        X[..., 1] += d
    elif c["shape"] == "bump":
        f = 0.1 * ly * np.exp(-((X[..., 0] - 0.5 * lx) ** 2) / (2.0 * 0.05 * (lx / 2) ** 2))
        X[..., 1] = X[..., 1] / ly * (ly - f) + f
    return X


def _lagrange(nodes, at):
    """(values, derivatives) [point][polynomial] of the Lagrange polynomials through `nodes`."""
    n = len(nodes)
    L, D = np.zeros((len(at), n)), np.zeros((len(at), n))
    for i in range(n):
        others = [nodes[j] for j in range(n) if j != i]
        den = np.prod([nodes[i] - o for o in others]) if others else 1.0
        for k, x in enumerate(at):
            L[k, i] = np.prod([x - o for o in others]) / den if others else 1.0
            D[k, i] = sum(np.prod([x - o for m, o in enumerate(others) if m != j]) for j in range(len(others))) / den
    return L, D


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _initial(c, seed, device):
    """The nodal state [E][5][nb], smooth fields drawn from the seed."""
    k, g = _constants(c), 1.4
    X = torch.tensor(_nodes(c), device=device).reshape(-1, *([c["q"] + 1] * 3), 3)
    P = c["p"] + 1
    r = np.arange(P) / c["p"] if c["p"] else np.zeros(1)
    L = torch.tensor(_lagrange(np.arange(c["q"] + 1) / c["q"], r)[0], device=device)
    x, y, z = torch.einsum("ck,bj,ai,ekjid->decba", L, L, L, X)
    lx, ly, lz = k["l"]
    rng = np.random.default_rng(seed)
    speed = {"tgv": 0.05, "fourier": 0.05, "channel": 0.05, "vortex": 0.0, "stream": 0.01}[c["flow"]]
    pert = [torch.zeros_like(x) for _ in range(4)]
    for f in range(4 if speed else 0):
        for _ in range(6):
            kx, ky, kz = (int(v) for v in rng.integers(1, 4, 3))
            amp, ph = speed / math.sqrt(6.0) * rng.standard_normal(), rng.uniform(0, TWO_PI, 3)
            pert[f] += amp * (torch.sin(TWO_PI * kx * x / lx + ph[0]) * torch.sin(TWO_PI * ky * y / ly + ph[1])
                              * torch.sin(TWO_PI * kz * z / lz + ph[2]))
    one = torch.ones_like(x)
    rho, pr = one * 1.0, one * (k["c"] ** 2 / g)
    u, v, w = one * k["u"] + pert[0], one * k["v"] + pert[1], one * k["w"] + pert[2]
    if c["flow"] == "tgv":
        sx, sy = x + rng.uniform(0, TWO_PI), y + rng.uniform(0, TWO_PI)
        u = u + torch.sin(sx) * torch.cos(sy) * torch.cos(z)
        v = v - torch.cos(sx) * torch.sin(sy) * torch.cos(z)
        pr = pr + (torch.cos(2 * sx) + torch.cos(2 * sy)) * (torch.cos(2 * z) + 2.0) / 16.0
        rho = pr / (k["c"] ** 2 / g)
    elif c["flow"] == "vortex":
        cx, cy = rng.uniform(4.0, 6.0, 2)
        r2 = (x - cx) ** 2 + (y - cy) ** 2
        e = 5.0 / TWO_PI * torch.exp(0.5 * (1 - r2))
        u, v = u - (y - cy) * e, v + (x - cx) * e
        T = 1.0 - (g - 1.0) * 25.0 / (8 * g * math.pi ** 2) * torch.exp(1 - r2)
        rho, pr = T ** (1 / (g - 1)), T ** (g / (g - 1))
    elif c["flow"] == "channel":
        s = 2.0 * y / ly - 1.0
        u = 1.5 * (1 - s * s) + pert[0] * (1 - s * s)
        v, w = v * (1 - s * s), w * (1 - s * s)
    else:
        rho = rho * (1 + 0.2 * pert[3])
    U = torch.stack([rho, rho * u, rho * v, rho * w, pr / (g - 1) + 0.5 * rho * (u * u + v * v + w * w)], 1)
    return U.reshape(U.shape[0], 5, -1).contiguous()


def _weights(c, seed, device):
    """A smooth-ish adjoint input: the gradient of an output functional in the state."""
    g = torch.Generator().manual_seed(seed * 7 + 1)
    n = 5 * (c["p"] + 1) ** 3
    return torch.randn(c["nx"] * c["ny"] * c["nz"], n, generator=g, dtype=torch.float64).to(device)


def _dt(c):
    k = _constants(c)
    h = min(k["l"][0] / c["nx"], k["l"][1] / c["ny"], k["l"][2] / c["nz"])
    return 0.15 * h / ((2 * c["p"] + 1) * (k["c"] + 1.5))


def prepare(case, seed):
    c, k = case, _constants(case)
    src = (0.0, k["src"], 0.0, 0.0, 0.0)
    prm = dg.make_reference_state(mu=k["mu"], c=k["c"], u=k["u"], v=k["v"], w=k["w"], source=src)
    mesh = dg.Mesh(c["nx"], c["ny"], c["nz"], c["p"], c["q"], _nodes(c), SIDES[c["sides"]])
    s = dg.Solver(mesh, prm, dg.MIXED_FP32 if c["precision"] == "mixed" else dg.FP64)
    if c["pr"]:
        s.set_prandtl(c["pr"])
    U = _initial(c, seed, "cuda").reshape(-1)
    st = {"case": c, "solver": s, "scheme": dg.TIME_SCHEMES[c["scheme"]], "dt": _dt(c), "U": U}
    if c["kind"] == "step":
        st["out"] = torch.empty_like(U)
    elif c["kind"] == "residual":
        st["R"], st["f"] = torch.empty_like(U), torch.empty_like(U)
    elif c["kind"] == "host":
        st["in"], st["out"] = U.cpu().pin_memory(), torch.empty(U.shape, dtype=U.dtype).pin_memory()
    else:
        st["U"] = U.requires_grad_()
        st["lam"] = _weights(c, seed, "cuda").reshape(-1)
        theta = [k["mu"], *src] + ([prm.T] if c["sides"] == "isothermal" else [])
        st["theta"] = torch.tensor(theta, dtype=torch.float64, requires_grad=True)
    torch.cuda.synchronize()
    return st


def run(st):
    c, s = st["case"], st["solver"]
    if c["kind"] == "step":
        s.set_state_device(st["U"].data_ptr())
        norms = s.step(st["scheme"], st["dt"], c["steps"])
        s.get_state_device(st["out"].data_ptr())
        return {"state": st["out"], "norms": norms}
    if c["kind"] == "host":
        norms = s.step_host(st["scheme"], st["dt"], c["steps"], st["in"].numpy(), st["out"].numpy())
        return {"state": st["out"], "norms": norms}
    if c["kind"] == "residual":
        s.residual_device(st["U"].data_ptr(), st["R"].data_ptr(), st["f"].data_ptr())
        s.synchronize()
        return {"R": st["R"], "f": st["f"]}
    if c["kind"] == "vjp":
        f = ag.residual(st["U"], s)
        (g,) = torch.autograd.grad(f, st["U"], st["lam"])
        return {"f": f.detach(), "grad": g}
    UN = ag.integrate(st["U"], s, st["scheme"], st["dt"], c["steps"], c["slots"], theta=st["theta"])
    g, gt = torch.autograd.grad(UN, (st["U"], st["theta"]), st["lam"])
    return {"state": UN.detach(), "grad": g, "grad_theta": gt}


# ------------------------------------------------------------------ the bytes and operations of a pass

def work(case):
    """Bytes: the state read and written once, the parts of the geometry that
    the element shape needs, and per RK stage what a fused stage cannot do
    without (its input, the step's base and the accumulator; TVD-RK3 has no
    accumulator).  Operations: the discretisation in sum-factorised form."""
    c = case
    E, P = c["nx"] * c["ny"] * c["nz"], c["p"] + 1
    nb, nqf = P ** 3, P * P
    curved = c["shape"] in ("sine", "bump")
    viscous = c["flow"] != "vortex"
    geo = 80.0 + ((80.0 * nb + 96.0 * nqf) if curved else 0.0)
    # gradients and tests 60 P^4, the pointwise flux, per face point traces, fluxes and tests
    stage = 60.0 * P ** 4 + nb * (230.0 if viscous else 70.0) + 6 * nqf * (20.0 * P + (350.0 if viscous else 130.0))
    stages = 4 if c["scheme"] == "RK4" else 3
    per_stage = (200.0 if stages == 4 else 120.0) * nb + geo
    state = 40.0 * nb
    if c["kind"] == "residual":
        return {"bytes": E * (3 * state + geo), "flops": E * (stage + 60.0 * P ** 4)}
    if c["kind"] == "vjp":
        return {"bytes": E * (2 * state + geo + 3 * state + geo), "flops": E * 3.5 * (stage + 60.0 * P ** 4)}
    n = c["steps"] * stages
    if c["kind"] == "adjoint":  # forward, and per reversed step its stages again and their transposes
        return {"bytes": E * n * (3.5 * per_stage), "flops": E * n * 4.5 * stage}
    return {"bytes": E * (n * per_stage + 2 * state), "flops": E * n * stage}


# ------------------------------------------------------------------ the same in plain torch float64

class _Plain:
    """The DG residual in the Gauss-point basis.  Arrays are [nz][ny][nx][...];
    a volume field ends in [z][y][x], a face field in [t2][t1] (t1 < t2)."""

    def __init__(self, c, mu, kq, src, Tw, device):
        self.c, self.mu, self.kq, self.src, self.Tw = c, mu, kq, src, Tw
        k = _constants(c)
        self.g, self.Rg, self.eta = 1.4, 287.0, 6.0
        P = c["p"] + 1
        x, w = np.polynomial.legendre.leggauss(P)
        x, w = 0.5 * (x + 1), 0.5 * w
        dd = dict(dtype=torch.float64, device=device)
        t = lambda a: torch.tensor(a, **dd)  # noqa: E731
        r = np.arange(P) / c["p"] if c["p"] else np.zeros(1)
        self.B = t(_lagrange(r, x)[0])
        self.Bi = t(np.linalg.inv(_lagrange(r, x)[0]))
        self.Dq, self.EL = t(_lagrange(x, x)[1]), t(_lagrange(x, [0.0, 1.0])[0])
        self.DL = t(_lagrange(x, [0.0, 1.0])[1])
        wt = t(w)
        self.w3, self.w2 = torch.einsum("a,b,c->abc", wt, wt, wt), torch.einsum("a,b->ab", wt, wt)
        gn = np.arange(c["q"] + 1) / c["q"]
        X = t(_nodes(c))

        def metrics(at):  # at = (x, y, z) points; d xi_i / d x_c [i][c] and the Jacobian
            LD = [[t(m) for m in _lagrange(gn, a)] for a in at]
            J = torch.stack([torch.einsum("az,by,cx,KJIzyxd->KJIabcd", LD[2][i == 2], LD[1][i == 1], LD[0][i == 0], X)
                             for i in range(3)], -1)  # [..., d, i] = d X_d / d xi_i
            inv = torch.linalg.inv(J)
            return inv.permute(6, 7, 0, 1, 2, 3, 4, 5), torch.linalg.det(J)

        self.Ji, self.dJ = metrics((x, x, x))
        self.face = []
        for lf in range(6):
            a, end = lf >> 1, lf & 1
            at = [x, x, x]
            at[a] = np.array([float(end)])
            Ji, dJ = metrics(at)
            ax = 5 - a  # the array axis of direction a in [K][J][I][z][y][x]
            Ji, dJ = Ji.squeeze(ax + 2), dJ.squeeze(ax)
            nv = Ji[a] * dJ * (1.0 if end else -1.0)
            fJ = nv.square().sum(0).sqrt()
            lift = torch.tensordot(1.0 / self.dJ, self.EL[end] ** 2 / wt, dims=([ax], [0]))
            self.face.append((Ji, nv / fJ, fJ, lift))
        # total conditions of the inflow, the outflow's pressure and the freestream
        v2 = k["u"] ** 2 + k["v"] ** 2 + k["w"] ** 2
        self.p0 = k["c"] ** 2 / self.g
        M2 = v2 / k["c"] ** 2
        T = self.p0 / self.Rg
        f = 1 + 0.5 * (self.g - 1) * M2
        self.Tt, self.Pt = T * f, self.p0 * f ** (self.g / (self.g - 1))
        self.free = [1.0, k["u"], k["v"], k["w"], self.p0 / (self.g - 1) + 0.5 * v2]

    # states are lists of the five conserved fields
    def prim(self, S):
        u = [S[1] / S[0], S[2] / S[0], S[3] / S[0]]
        p = (self.g - 1) * (S[4] - 0.5 * S[0] * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))
        return u, p

    def euler_n(self, S, n):
        u, p = self.prim(S)
        m = S[0] * (u[0] * n[0] + u[1] * n[1] + u[2] * n[2])
        return [m, m * u[0] + p * n[0], m * u[1] + p * n[1], m * u[2] + p * n[2], m * (S[4] + p) / S[0]]

    def visc(self, S, G):
        """Q[c][r] = A(S, G), G[c][r] = d S_r / d x_c, with the heat flux."""
        u, _ = self.prim(S)
        du = [[(G[c][1 + i] - G[c][0] * u[i]) / S[0] for c in range(3)] for i in range(3)]
        div = du[0][0] + du[1][1] + du[2][2]
        Q = []
        for c in range(3):
            tau = [self.mu * (du[i][c] + du[c][i]) - (2.0 / 3.0 * self.mu * div if i == c else 0.0) for i in range(3)]
            e = u[0] * tau[0] + u[1] * tau[1] + u[2] * tau[2]
            eT = (G[c][4] - S[4] / S[0] * G[c][0]) / S[0] - sum(u[i] * du[i][c] for i in range(3))
            Q.append([torch.zeros_like(e), tau[0], tau[1], tau[2], e + self.kq * eT])
        return Q

    def rank1(self, S, d, n):
        return self.visc(S, [[d[r] * n[c] for r in range(5)] for c in range(3)])

    def normal(self, Q, n):
        return [Q[0][r] * n[0] + Q[1][r] * n[1] + Q[2][r] * n[2] for r in range(5)]

    def roe(self, L, R, n):
        g1 = self.g - 1
        (uL, pL), (uR, pR) = self.prim(L), self.prim(R)
        HL, HR = (L[4] + pL) / L[0], (R[4] + pR) / R[0]
        sL, sR = L[0].sqrt(), R[0].sqrt()
        u = [(sL * uL[i] + sR * uR[i]) / (sL + sR) for i in range(3)]
        H = (sL * HL + sR * HR) / (sL + sR)
        q2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        a = (g1 * (H - 0.5 * q2)).sqrt()
        un = u[0] * n[0] + u[1] * n[1] + u[2] * n[2]
        eps = 0.05 * a

        def fix(v):
            return torch.where(v.abs() < eps, ((eps * eps + v * v) / (2 * eps)).abs(), v.abs())

        a1, a2, a3 = fix(un + a), fix(un - a), fix(un)
        d = [R[r] - L[r] for r in range(5)]
        s1, s2 = 0.5 * (a1 + a2), 0.5 * (a1 - a2)
        G1 = g1 * (0.5 * q2 * d[0] - (u[0] * d[1] + u[1] * d[2] + u[2] * d[3]) + d[4])
        G2 = -un * d[0] + (d[1] * n[0] + d[2] * n[1] + d[3] * n[2])
        C1 = G1 / (a * a) * (s1 - a3) + G2 / a * s2
        C2 = G1 / a * s2 + (s1 - a3) * G2
        diss = [a3 * d[0] + C1] + [a3 * d[1 + i] + C1 * u[i] + C2 * n[i] for i in range(3)] + [a3 * d[4] + C1 * H + C2 * un]
        FL, FR = self.euler_n(L, n), self.euler_n(R, n)
        return [0.5 * (FL[r] + FR[r] - diss[r]) for r in range(5)]

    def ghost(self, bt, S, n):
        one, g, g1 = torch.ones_like(S[0]), self.g, self.g - 1
        if bt == FREE:
            return [one * v for v in self.free]
        if bt in (NOSLIP, ISO):
            zero = 0.0 * one
            return [S[0], zero, zero, zero, S[4] if bt == NOSLIP else S[0] * (self.Rg / g1) * self.Tw]
        u, p = self.prim(S)
        un = u[0] * n[0] + u[1] * n[1] + u[2] * n[2]
        if bt == WALL:
            return [S[0]] + [S[0] * (u[i] - un * n[i]) for i in range(3)] + [S[4]]
        J = un + 2 * (g * p / S[0]).sqrt() / g1
        if bt == INFLOW:
            RT = g * self.Rg * self.Tt
            A, Bq, C = RT - 0.5 * g1 * J * J, -4 * RT / g1, 4 * RT / g1 ** 2 - J * J
            disc = (Bq * Bq - 4 * A * C).sqrt()
            s0, s1 = (-Bq + disc) / (2 * A), (-Bq - disc) / (2 * A)
            M = torch.where((s0 >= 0) & (s1 >= 0), torch.minimum(s0, s1), torch.where(s0 >= 0, s0, s1))
            T = self.Tt / (1 + 0.5 * g1 * M * M)
            pb = self.Pt * (T / self.Tt) ** (g / g1)
            rb = pb / (self.Rg * T)
            vb = -M * (g * pb / rb).sqrt()
            return [rb] + [rb * vb * n[i] for i in range(3)] + [pb / g1 + 0.5 * rb * vb * vb]
        rb = (self.p0 / (p / S[0] ** g)) ** (1 / g)
        ub = J - 2 * (g * self.p0 / rb).sqrt() / g1
        v = [u[i] + (ub - un) * n[i] for i in range(3)]
        return [rb] + [rb * v[i] for i in range(3)] + [self.p0 / g1 + 0.5 * rb * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)]

    def along(self, M, S, a):
        """M contracted with direction a (0: x) of fields [..., z, y, x]."""
        return torch.einsum(("pk,...zyk->...zyp", "pk,...zkx->...zpx", "pk,...kyx->...pyx")[a], M, S)

    def residual(self, V):
        """Y and f_V = -Y / (w detJ) for Gauss-point values V[K][J][I][5][z][y][x]."""
        mu_on = not (isinstance(self.mu, float) and self.mu == 0.0)
        S = V.unbind(3)
        ref = [self.along(self.Dq, V, i).unbind(3) for i in range(3)]
        G = [[sum(self.Ji[i][c] * ref[i][r] for i in range(3)) for r in range(5)] for c in range(3)]
        u, p = self.prim(S)
        H = []
        for c in range(3):
            m = S[0] * u[c]
            F = [m, m * u[0], m * u[1], m * u[2], m * (S[4] + p) / S[0]]
            F[1 + c] = F[1 + c] + p
            H.append([-f for f in F])
        if mu_on:
            Q = self.visc(S, G)
            H = [[H[c][r] + Q[c][r] for r in range(5)] for c in range(3)]
        wJ = self.w3 * self.dJ
        Y = 0
        for i in range(3):
            C = torch.stack([wJ * sum(self.Ji[i][c] * H[c][r] for c in range(3)) for r in range(5)], 3)
            Y = Y + self.along(self.Dq.T, C, i)
        Y = Y - torch.stack([s * wJ for s in self.src], 3)
        # face traces: values and viscous normal flux
        tr = []
        for lf in range(6):
            a, end = lf >> 1, lf & 1
            line = ("k,...zyk->...zy", "k,...zkx->...zx", "k,...kyx->...yx")[a]
            St = torch.einsum(line, self.EL[end], V)
            t1, t2 = [d for d in range(3) if d != a]
            g = [None] * 3
            g[a] = torch.einsum(line, self.DL[end], V)
            g[t1] = torch.einsum("pk,...tk->...tp", self.Dq, St)
            g[t2] = torch.einsum("pk,...kt->...pt", self.Dq, St)
            Ji, n, fJ, lift = self.face[lf]
            Sl, Qn = St.unbind(3), None
            if mu_on:
                gl = [q.unbind(3) for q in g]
                Gf = [[sum(Ji[i][c] * gl[i][r] for i in range(3)) for r in range(5)] for c in range(3)]
                Qn = self.normal(self.visc(Sl, Gf), n)
            tr.append((Sl, Qn))
        for lf in range(6):
            a, end = lf >> 1, lf & 1
            ax, bt = 2 - a, SIDES[self.c["sides"]][lf]
            N = V.shape[ax]
            Ji, n, fJ, lift = self.face[lf]

            def other(f):  # the neighbour's field across this face (wrapped)
                return torch.roll(f, -1 if end else 1, ax)

            parts = [(None, 0, N)] if bt == PER else (
                [(None, 0, N - 1), (bt, N - 1, 1)] if end else [(bt, 0, 1), (None, 1, N - 1)])
            done = []
            for kind, s0, ln in parts:
                if ln == 0:
                    continue
                cut = lambda f: f.narrow(ax, s0, ln)  # noqa: E731,B023
                Uo, nn, fj, lo = [cut(f) for f in tr[lf][0]], [cut(f) for f in n], cut(fJ), cut(lift)
                Qo = [cut(f) for f in tr[lf][1]] if mu_on else None
                if kind is None:
                    Un = [cut(other(f)) for f in tr[lf ^ 1][0]]
                    fa = self.roe(Uo, Un, nn)
                    jump, dual = [x - y for x, y in zip(Uo, Un)], 0.5
                    if mu_on:
                        Qx = [cut(other(f)) for f in tr[lf ^ 1][1]]
                        ro, rn = (self.normal(self.rank1(s, jump, nn), nn) for s in (Uo, Un))
                        ln_ = cut(other(self.face[lf ^ 1][3]))
                        fa = [fa[r] - 0.5 * (Qo[r] - Qx[r]) + 0.25 * self.eta * fj * (lo * ro[r] + ln_ * rn[r])
                              for r in range(5)]
                else:
                    Ub = self.ghost(kind, Uo, nn)
                    fa = self.euler_n(Ub, nn)
                    jump, dual = [x - y for x, y in zip(Uo, Ub)], 1.0
                    if mu_on:
                        rb = self.normal(self.rank1(Ub, jump, nn), nn)
                        fa = [fa[r] - Qo[r] + self.eta * fj * lo * rb[r] for r in range(5)]
                fw = fj * self.w2
                fa = [f * fw for f in fa]
                fb = None
                if mu_on:
                    dc = self.rank1(Uo, [dual * j for j in jump], nn)
                    Jc = [[cut(Ji[i][c]) for c in range(3)] for i in range(3)]
                    fb = [torch.stack([-fw * sum(Jc[i][c] * dc[c][r] for c in range(3)) for r in range(5)], 3)
                          for i in range(3)]
                done.append((torch.stack(fa, 3), fb))
            fa = torch.cat([d[0] for d in done], ax)
            t1, t2 = [d for d in range(3) if d != a]
            out = ("k,...zy->...zyk", "k,...zx->...zkx", "k,...yx->...kyx")[a]
            if mu_on:
                fb = [torch.cat([d[1][i] for d in done], ax) for i in range(3)]
                fa = fa + torch.einsum("kp,...tk->...tp", self.Dq, fb[t1]) + torch.einsum("kp,...kt->...pt", self.Dq, fb[t2])
                Y = Y + torch.einsum(out, self.DL[end], fb[a])
            Y = Y + torch.einsum(out, self.EL[end], fa)
        return Y, -Y / wJ[:, :, :, None]

    def basis(self, M, U):
        for a in range(3):
            U = self.along(M, U, a)
        return U

    def step(self, V, dt, scheme):
        Y, k1 = self.residual(V)
        if scheme == "RK4":
            k2 = self.residual(V + 0.5 * dt * k1)[1]
            k3 = self.residual(V + 0.5 * dt * k2)[1]
            k4 = self.residual(V + dt * k3)[1]
            return V + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4), Y
        V1 = V + dt * k1
        V2 = 0.75 * V + 0.25 * V1 + 0.25 * dt * self.residual(V1)[1]
        return V / 3.0 + 2.0 / 3.0 * V2 + 2.0 / 3.0 * dt * self.residual(V2)[1], Y


def exact(case, seed):
    c, dev = case, _device()
    E, P = c["nx"] * c["ny"] * c["nz"], c["p"] + 1
    stages = c["steps"] * (4 if c["scheme"] == "RK4" else 3) if c["kind"] in ("step", "host", "adjoint") else 1
    cost = 5.0 * E * P ** 3 * stages * (8 if c["kind"] in ("adjoint", "vjp") else 1)
    if cost > (1.5e9 if dev == "cuda" else 4e6):
        return None
    k = _constants(c)
    leaf = [k["mu"], 0.0, k["src"], 0.0, 0.0, 0.0, k["c"] ** 2 / 1.4 / 287.0]  # mu, the five sources, Tw
    theta = [torch.tensor(v, dtype=torch.float64, device=dev) for v in leaf]
    grad = c["kind"] in ("vjp", "adjoint")
    if c["kind"] == "adjoint":
        theta = [t.requires_grad_() for t in theta]
    mu = theta[0] if k["mu"] or c["kind"] == "adjoint" else 0.0
    kq = mu * 1.4 / c["pr"] if c["pr"] else 0.0
    U = _initial(c, seed, dev).reshape(c["nz"], c["ny"], c["nx"], 5, P, P, P)
    U.requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        D = _Plain(c, mu, kq, theta[1:6], theta[6], dev)
        nodal = lambda A: D.basis(D.Bi, A)  # noqa: E731
        if c["kind"] == "residual" or c["kind"] == "vjp":
            Y, f = D.residual(D.basis(D.B, U))
            f = nodal(f).reshape(-1)
            if c["kind"] == "residual":
                return {"R": D.basis(D.B.T, Y).reshape(-1), "f": f}
            (g,) = torch.autograd.grad(f, U, _weights(c, seed, dev).reshape(-1))
            return {"f": f.detach(), "grad": g.reshape(-1)}
        V = D.basis(D.B, U.detach())
        states, norms = [], []
        with torch.no_grad():
            for _ in range(c["steps"]):
                states.append(V)
                V, Y = D.step(V, _dt(c), c["scheme"])
                norms.append(float(D.basis(D.B.T, Y).square().mean().sqrt()))
            last = nodal(V).reshape(-1)
        if c["kind"] != "adjoint":
            return {"state": last, "norms": np.array(norms)}
        lam = D.basis(D.Bi.T, _weights(c, seed, dev).reshape(U.shape))  # dJ/dV from dJ/dU
        gt = [torch.zeros((), dtype=torch.float64, device=dev) for _ in theta]
        for V in reversed(states):
            V = V.detach().requires_grad_()
            VN, _ = D.step(V, _dt(c), c["scheme"])
            got = torch.autograd.grad(VN, [V, *theta], lam, allow_unused=True, retain_graph=True)
            lam, gt = got[0], [a + b if b is not None else a for a, b in zip(gt, got[1:])]
            del VN, got
        n = 7 if c["sides"] == "isothermal" else 6
        return {"state": last, "grad": D.basis(D.B.T, lam).reshape(-1),
                "grad_theta": torch.stack(gt)[:n].cpu()}
