"""Performance cases: the work a program hands to this library, with sizes.

A case is one frame interval of the host driver's loop (`scp_sim`): steps in
runs of the diagnostics cadence, a diagnostics row after each run, and one
snapshot of every column at the end, copied to page-locked host memory while
the next interval may already step (`snapshot_async`, which waits for the
previous frame of the same handle).  A further kind stands for the begin of a
run: `start`, a handle made from host columns, its first diagnostics row and
frame.

Every kind has `exact`, a restatement in plain torch (complex128 matter
fields, float64 links) of the same equations: fused kick / drift / kick
leapfrog, covariant stencils, start-up Gauss projection by Fourier transform,
and the diagnostics.  Inputs depend on the seed alone.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from scp_b200.api import DTYPE_F32, DTYPE_F64, Simulation
from scp_b200.params import DIAG_NAMES, PREC_FP32C, PREC_FP64, Params

DT = torch.float64
KINDS = ("complex", "gauged", "sponge", "higgs", "fabrics", "real")


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest grid in use: every call is launches and latency
        dict(name="gauged_32", kind="gauged", n=32, steps=50, every=10, fp32c=False, frame64=True),
        # the ungauged model at the 64^3 size of the simplest workload (state near the L2 size)
        dict(name="complex_64", kind="complex", n=64, steps=100, every=10, fp32c=False, frame64=True),
        # odd edge with the absorbing sponge: ragged tiles in both directions, single-precision frames
        dict(name="sponge_97", kind="sponge", n=97, steps=100, every=10, fp32c=False, frame64=False),
        # the flagship: two opposite balls in the gauged model at 128^3, checkpoint frames
        dict(name="gauged_128", kind="gauged", n=128, steps=200, every=10, fp32c=False, frame64=True),
        # the same model at production size
        dict(name="gauged_256", kind="gauged", n=256, steps=100, every=25, fp32c=False, frame64=False),
        # the compensated single-precision mode at production size
        dict(name="gauged_256_fp32c", kind="gauged", n=256, steps=100, every=25, fp32c=True, frame64=False),
        # the compensated mode on an odd edge (one site per thread)
        dict(name="gauged_95_fp32c", kind="gauged", n=95, steps=100, every=10, fp32c=True, frame64=False),
        # the ungauged model in the compensated mode, edge not a power of two
        dict(name="complex_200_fp32c", kind="complex", n=200, steps=100, every=25, fp32c=True, frame64=False),
        # Higgs condensate and second gauge
        dict(name="higgs_128", kind="higgs", n=128, steps=50, every=10, fp32c=False, frame64=True),
        # three matter fabrics, Q locked to C
        dict(name="fabrics_128", kind="fabrics", n=128, steps=50, every=10, fp32c=False, frame64=False),
        # the real six-field model with its optional force terms
        dict(name="real_128", kind="real", n=128, steps=100, every=10, fp32c=False, frame64=True),
        # start of a run: upload, net-charge check, Gauss projection, first row and frame
        dict(name="start_96", kind="start", n=96, steps=0, every=0, fp32c=False, frame64=True),
    ]


def draw(rng):
    """One more case: any kind, edges spread over their logarithm (odd ones
    among them), steps and cadence bounded so that it stays below the largest."""
    if rng.random() < 0.1:
        fp32c = rng.random() < 0.5
        return dict(kind="start", n=int(round(math.exp(rng.uniform(math.log(24), math.log(144))))), steps=0, every=0,
                    fp32c=fp32c, frame64=not fp32c)
    kind = rng.choice(KINDS + ("gauged",))
    n = int(round(math.exp(rng.uniform(math.log(24), math.log(200)))))
    every = rng.choice((10, 10, 20, 25))
    most = min(8, max(1, int(4e8 / n ** 3) // every))
    fp32c = kind in ("complex", "gauged", "sponge") and rng.random() < 0.4
    return dict(kind=kind, n=n, steps=every * rng.randint(1, most), every=every, fp32c=fp32c,
                frame64=not fp32c and rng.random() < 0.5)


def params_of(case) -> Params:
    """Lattice spacing 0.5 and time step 0.1, as the repository's workloads."""
    n, kind = case["n"], case["kind"]
    kw = dict(N=n, L=(n - 1) / 4.0, dt_factor=0.2, bc_type=2, precision=PREC_FP32C if case["fp32c"] else PREC_FP64)
    if kind in ("gauged", "start"):
        kw.update(complex_gauge=1, g_gauge=0.1)
    elif kind == "sponge":
        kw.update(complex_gauge=1, g_gauge=0.1, bc_type=0, damp_width=min(3.0, 0.2 * (n - 1) / 4.0), damp_rate=0.01)
    elif kind == "higgs":
        kw.update(complex_gauge=1, g_gauge=0.1, higgs_v=1.0, higgs_rvoid=4.0, g_gauge2=0.1)
    elif kind == "fabrics":
        kw.update(complex_gauge=1, g_gauge=0.1, n_fabrics=3, mf_lock_CQ=1, q_C=0.0, q_Q=1.0, q_L=-1.0)
    elif kind == "real":
        kw.update(real_fields=1, mode=3, kappa_gamma=2.0, alpha_cs=0.1, beta_h=0.05, kappa_h=0.002)
    return Params(**kw)


# ---------------------------------------------------------------- inputs

def device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def noise(gen, shape, var):
    return torch.randn(shape, generator=gen, dtype=DT, device=gen.device) * math.sqrt(var)


def axes(p):
    x = -p.L + torch.arange(p.N, dtype=DT, device=device()) * p.dx
    return x[:, None, None], x[None, :, None], x[None, None, :]


def matter(p, seed, opposite=True):
    """Two Gaussian balls of opposite charge (component phases 2 pi a / 3) near
    x = -+5, moved and turned by the seed, with thermal noise on every field
    and the net charge removed: complex fields and velocities (6, N, N, N)."""
    rnd = random.Random(seed)
    gen = torch.Generator(device=device())
    gen.manual_seed(seed)
    X, Y, Z = axes(p)
    F = torch.complex(noise(gen, (6, p.N, p.N, p.N), 1e-3), noise(gen, (6, p.N, p.N, p.N), 1e-3))
    V = torch.zeros_like(F)
    off, sig = min(5.0, 0.4 * p.L), min(3.0, 0.25 * p.L)
    for sign in (-1.0, 1.0):
        cx, cy, cz = (sign * off if d == 0 else 0.0 for d in range(3))
        cx, cy, cz = (c + rnd.uniform(-0.5, 0.5) for c in (cx, cy, cz))
        env = torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2) / (2 * sig * sig))
        omega, turn = (sign if opposite else 1.0) * rnd.uniform(0.7, 0.9), rnd.uniform(0, 2 * math.pi)
        for a in range(3):
            ball = env * complex(math.cos(2 * math.pi * a / 3 + turn), math.sin(2 * math.pi * a / 3 + turn))
            F[a] += ball
            V[a] += 1j * omega * ball
    V += torch.complex(noise(gen, F.shape, 1e-4), noise(gen, F.shape, 1e-4))
    eps = -rho_of(F, V).sum() / F[:3].abs().square().sum()
    V[:3] += 1j * eps * F[:3]
    return F, V


def inputs(case, seed):
    """Everything a run of the case starts from, as named tensors."""
    p = params_of(case)
    shape = (3, p.N, p.N, p.N)
    if case["kind"] == "real":
        gen = torch.Generator(device=device())
        gen.manual_seed(seed)
        rnd = random.Random(seed)
        X, Y, Z = axes(p)
        f, v = torch.cat((torch.zeros(shape, dtype=DT, device=gen.device), noise(gen, shape, 1e-3))), noise(
            gen, (6,) + shape[1:], 1e-3)
        sig = min(3.0, 0.25 * p.L)
        for sign in (-1.0, 1.0):
            env = torch.exp(-((X - sign * 0.3 * p.L) ** 2 + Y ** 2 + Z ** 2) / (2 * sig * sig))
            for a in range(3):
                amp = rnd.uniform(0.6, 0.8)
                f[a] += amp * env
                v[a] -= 0.3 * amp * env
        return dict(f=f, v=v)
    F, V = matter(p, seed)
    got = dict(F=F, V=V)
    if p.complex_gauge:
        gen = torch.Generator(device=device())
        gen.manual_seed(seed + 1)
        got["th"] = noise(gen, shape, 0.01)
        got["E"] = noise(gen, shape, 1e-4)
    if case["kind"] == "fabrics":
        got["FL"], got["VL"] = matter(p, seed + 2)
    return got


def split(F):
    """SFA order of one multiplet's columns: u, tu of the fields."""
    return [F[a].real for a in range(6)], [F[a].imag for a in range(6)]


def columns(p, s):
    """The state's SFA columns, a list of (N, N, N) tensors."""
    if p.real_fields:
        return list(s["f"]) + list(s["v"])

    def multiplet(F, V):
        re, im = split(F)
        dre, dim = split(V)
        return re + dre + im + dim

    cols = multiplet(s["F"], s["V"])
    if p.complex_gauge:
        cols += list(s["th"]) + list(s["E"])
    if "th2" in s:
        cols += list(s["th2"]) + list(s["E2"])
    if "FL" in s:
        cols += multiplet(s["FL"], s["VL"])
    return cols


def host_columns(p, s):
    """Page-locked host columns as numpy arrays (fabric Q's, which a locked run
    ignores, stand between C's and L's)."""
    cols = columns(p, s)
    if "FL" in s:
        cols = cols[:30] + cols[:24] + cols[30:]
    host = torch.empty((len(cols), p.N ** 3), dtype=DT, pin_memory=torch.cuda.is_available())
    for h, c in zip(host, cols):
        h.copy_(c.reshape(-1))
    return list(host.numpy())


# ---------------------------------------------------------------- what is timed

def prepare(case, seed):
    p = params_of(case)
    cols = host_columns(p, inputs(case, seed))
    out = torch.empty((p.snap_ncols, p.N ** 3), dtype=torch.float64 if case["frame64"] else torch.float32,
                      pin_memory=torch.cuda.is_available())
    state = dict(case=case, out=list(out.numpy()), p=p)
    if case["kind"] == "start":
        state["cols"] = cols
    else:
        state["sim"] = Simulation(p, cols)
    return state


def table(case, rows):
    """Diagnostics rows; those of a compensated single-precision run are good to single precision."""
    return np.stack(rows).astype(np.float32 if case["fp32c"] else np.float64)


def run(state):
    case = state["case"]
    dtype = DTYPE_F64 if case["frame64"] else DTYPE_F32
    if case["kind"] == "start":
        with Simulation(state["p"], state["cols"]) as sim:
            row = table(case, [sim.diag_vector()])
            return dict(rows=row, frame=sim.snapshot(dtype, out=state["out"]))
    sim = state["sim"]
    rows = []
    for _ in range(case["steps"] // case["every"]):
        sim.step(case["every"])
        rows.append(sim.diag_vector())
    sim.snapshot_async(state["out"], dtype)
    return dict(rows=table(case, rows), frame=state["out"])


# words of state per site, and floating-point operations per site and step
# (transports, Laplacians, curls, currents, link phases and plaquettes)
WORDS = {"complex": 24, "gauged": 30, "sponge": 30, "start": 30, "higgs": 38, "fabrics": 54, "real": 12}
FLOPS = {"complex": 350, "gauged": 1500, "sponge": 1500, "start": 0, "higgs": 2800, "fabrics": 2700, "real": 400}


def work(case):
    kind, n3 = case["kind"], case["n"] ** 3
    words = WORDS[kind]
    # compensated mode: fp32 momenta, fp32 + bf16 matter positions, fp32 pairs of link angles
    state = 8 * words if not case["fp32c"] else (156 if kind != "complex" else 120)
    frame = n3 * words * (8 if case["frame64"] else 4)
    if kind == "start":   # columns up, both position buffers and momenta written, frame down
        return {"bytes": 8 * 30 * n3 + 2 * state * n3 + frame, "flops": 300.0 * n3}
    rows = case["steps"] // case["every"]
    return {"bytes": case["steps"] * 2 * state * n3 + rows * state * n3 + frame,
            "flops": float(case["steps"] + rows) * FLOPS[kind] * n3}


# ---------------------------------------------------------------- plain torch

def fwd(f, d):
    """f at x + d (d counts the three lattice axes)."""
    return torch.roll(f, -1, dims=d - 3)


def back(f, d):
    return torch.roll(f, 1, dims=d - 3)


def im_prod(a, b):
    """Im[a* b]."""
    return a.real * b.imag - a.imag * b.real


def rho_of(F, V):
    return im_prod(F, V).sum(0)


def div(E, dx):
    return sum(E[d] - back(E[d], d) for d in range(3)) / dx


def project(E, rho, g, dx):
    """One-time Gauss projection: E gains grad chi with lap chi = mean(G) - G."""
    n = E.shape[-1]
    G = div(E, dx) - g * rho
    k = (4 / dx ** 2) * torch.sin(math.pi * torch.arange(n, dtype=DT, device=E.device) / n) ** 2
    lam = k[:, None, None] + k[None, :, None] + k[None, None, :]
    lam[0, 0, 0] = 1.0
    chi = torch.fft.fftn(G - G.mean()) / lam
    chi[0, 0, 0] = 0.0
    chi = torch.fft.ifftn(chi).real
    E = torch.stack([E[d] + (fwd(chi, d) - chi) / dx for d in range(3)])
    return E, (div(E, dx) - g * rho).mean()


def curl(D, f0):
    """Curl of the 3-vector in fields f0..f0+2 from the central differences D[d]."""
    return torch.stack([D[(a + 1) % 3][f0 + (a + 2) % 3] - D[(a + 2) % 3][f0 + (a + 1) % 3] for a in range(3)])


def plaquettes(th, fn):
    return [fn(th[a] + fwd(th[b], a) - fwd(th[a], b) - th[b]) for a, b in ((0, 1), (1, 2), (2, 0))]


def staples(th):
    p0, p1, p2 = plaquettes(th, torch.sin)
    return torch.stack(((p0 - back(p0, 1)) - (p2 - back(p2, 2)), (p1 - back(p1, 2)) - (p0 - back(p0, 0)),
                        (p2 - back(p2, 0)) - (p1 - back(p1, 1))))


def transports(F, U):
    """Forward and backward transports per direction (U[d]: link phases, or None)."""
    if U is None:
        return [fwd(F, d) for d in range(3)], [back(F, d) for d in range(3)]
    return [U[d] * fwd(F, d) for d in range(3)], [back(U[d].conj() * F, d) for d in range(3)]


def matter_force(p, F, U, W, weights=None):
    """Accelerations of one multiplet, its lattice current per direction and,
    with weights, the weighted one.  W[d]: link phase of the cross term."""
    idx1, idx2 = 1 / (2 * p.dx), 1 / p.dx ** 2
    Tp, Tm = transports(F, U)
    lap = (sum(Tp) + sum(Tm) - 6 * F) * idx2
    D = [(a - b) * idx1 for a, b in zip(Tp, Tm)]
    s = F[:3].abs().square()
    rest = torch.stack((s[1] * s[2], s[0] * s[2], s[0] * s[1]))
    prod = s[0] * rest[0]
    acc = lap
    acc[:3] += -p.m2 * F[:3] - (p.mu / (1 + p.kappa * prod) ** 2) * rest * F[:3] + p.eta * curl(D, 3)
    acc[3:] += -p.mtheta2 * F[3:] + p.eta * curl(D, 0)
    if U is None:
        return acc, None, None
    J, Jw = [], []
    for d in range(3):
        per = im_prod(F, Tp[d])
        d1, d2 = (d + 1) % 3, (d + 2) % 3
        theta = fwd(F[3:], d)
        Wphi = W[d].conj() * F[:3]
        cross = [im_prod(F[3 + e], Tp[d][f]) + im_prod(theta[e], Wphi[f]) for e, f in ((d1, d2), (d2, d1))]
        J.append(per.sum(0) / p.dx - 0.5 * p.eta * (cross[0] - cross[1]))
        if weights is not None:
            Jw.append(sum(w * (per[a] + per[3 + a]) for a, w in enumerate(weights)) / p.dx)
    return acc, torch.stack(J), torch.stack(Jw) if Jw else None


class Plain:
    """The same run in plain torch, 64 bits throughout."""

    def __init__(self, p, s):
        self.p, self.s = p, {k: v.clone() for k, v in s.items()}
        s, self.offset = self.s, 0.0
        dev = device()
        if p.gauge2:
            s["th2"], s["E2"] = torch.zeros_like(s["th"]), torch.zeros_like(s["E"])
        if p.higgs_v > 0 and p.complex_gauge:
            X, Y, Z = axes(p)
            r = torch.sqrt(X * X + Y * Y + Z * Z)
            s["H"] = p.higgs_v * 0.5 * (1 + torch.tanh((r - p.higgs_rvoid) / 0.6)) if p.higgs_rvoid > 0 else \
                torch.full_like(r, p.higgs_v)
            s["Hd"] = torch.zeros_like(s["H"])
        self.charges = (p.gauge2_q0, p.gauge2_q1, p.gauge2_q2)
        if p.gauged:
            s["E"], self.offset = project(s["E"], self.rho_em(), p.g_gauge, p.dx)
        if p.gauge2:
            per = im_prod(s["F"], s["V"])
            rho2 = sum(q * (per[a] + per[3 + a]) for a, q in enumerate(self.charges))
            s["E2"], _ = project(s["E2"], rho2, p.g_gauge2, p.dx)
        self.damp = None
        if p.bc_type == 0 and p.damp_width > 0 and p.damp_rate > 0:
            X, Y, Z = axes(p)
            r = torch.sqrt(X * X + Y * Y + Z * Z)
            t = ((r - (p.L - p.damp_width)) / p.damp_width).clamp(0, 1)
            self.damp = 1 - p.damp_rate * t * t
        self.dev = dev
        self.acc = self.force()

    def rho_em(self):
        s, p = self.s, self.p
        if "FL" in s:
            c = rho_of(s["F"], s["V"])
            return (p.q_C + p.q_Q) * c + p.q_L * rho_of(s["FL"], s["VL"])
        return rho_of(s["F"], s["V"])

    def links(self, q=1.0):
        th = q * self.s["th"]
        return torch.polar(torch.ones_like(th), th)

    def force(self):
        """Accelerations by momentum name."""
        p, s = self.p, self.s
        if p.real_fields:
            return {"v": self.real_force()}
        if not p.gauged:
            return {"V": matter_force(p, s["F"], None, None)[0]}
        stp = 1 / (p.g_gauge * p.dx ** 3)
        if p.n_fabrics == 3:   # C moves under the locked Q's force; both add their currents
            U = self.links(p.q_Q)
            a, J, _ = matter_force(p, s["F"], U, U)
            K = stp * staples(s["th"]) + p.g_gauge * p.q_Q * J
            if p.q_C != 0:
                UC = self.links(p.q_C)
                K = K + p.g_gauge * p.q_C * matter_force(p, s["F"], UC, UC)[1]
            UL = self.links(p.q_L)
            aL, JL, _ = matter_force(p, s["FL"], UL, UL)
            return {"V": a, "VL": aL, "E": K + p.g_gauge * p.q_L * JL}
        U = W = self.links()
        weights = None
        if p.gauge2:
            weights = self.charges
            ph = torch.stack([s["th"] + q * s["th2"] for q in weights], 1)
            U = torch.polar(torch.ones_like(ph), ph).repeat(1, 2, 1, 1, 1)
        a, J, Jw = matter_force(p, s["F"], U, W, weights)
        got = {"V": a, "E": stp * staples(s["th"]) + p.g_gauge * J}
        if p.gauge2:
            got["E2"] = staples(s["th2"]) / (p.g_gauge2 * p.dx ** 3) + p.g_gauge2 * Jw
        if "H" in s:
            H, sq = s["H"], s["F"][:3].abs().square()
            prod = sq[0] * sq[1] * sq[2]
            rest = torch.stack((sq[1] * sq[2], sq[0] * sq[2], sq[0] * sq[1]))
            a[:3] -= p.higgs_kap * H * H * rest * s["F"][:3]
            lap = (sum(fwd(H, d) + back(H, d) for d in range(3)) - 6 * H) / p.dx ** 2
            got["Hd"] = lap - p.higgs_lam * H * (H * H - p.higgs_v ** 2) - p.higgs_kap * prod * H
        return got

    def grads(self, f):
        return [(fwd(f, d) - back(f, d)) / (2 * self.p.dx) for d in range(3)]

    def real_force(self):
        p, f = self.p, self.s["f"]
        phi, th = f[:3], f[3:]
        D = self.grads(f)
        cp, ct = curl(D, 0), curl(D, 3)
        lap = (sum(fwd(f, d) + back(f, d) for d in range(3)) - 6 * f) / p.dx ** 2
        sig = phi.square().sum(0)
        m2 = p.inv_alpha / (1 + p.inv_beta * sig) if p.mode == 1 else p.m2
        ke = p.kappa / (1 + p.kappa_gamma * sig) if p.mode == 3 else p.kappa
        P = phi[0] * phi[1] * phi[2]
        P2 = P * P
        dP = torch.stack((phi[1] * phi[2], phi[2] * phi[0], phi[0] * phi[1]))
        acc = lap
        acc[:3] += -m2 * phi - (p.mu * P / (1 + ke * P2) ** 2) * dP + p.eta * ct
        if p.mode == 3 and p.kappa_gamma > 0:
            den = 1 + p.kappa_gamma * sig + p.kappa * P2
            acc[:3] -= (p.mu * p.kappa_gamma * p.kappa * P2 * P2 / den ** 2) * phi
        if p.kappa_h != 0:
            hel = (phi * cp).sum(0)
            acc[:3] += p.kappa_h * (2 * P * hel * dP + 2 * P2 * cp +
                                    torch.linalg.cross(torch.stack(self.grads(P2)), phi, dim=0))
        acc[3:] += -p.mtheta2 * th + p.eta * cp - p.beta_h * cp.square().sum(0) * th
        if p.alpha_cs != 0:
            C = 0.5 * cp - th
            acc[:3] -= p.alpha_cs * curl(self.grads(C), 0)
            acc[3:] += 2 * p.alpha_cs * C
        if p.beta_h != 0:
            acc[:3] -= 2 * curl(self.grads(0.5 * p.beta_h * th.square().sum(0) * cp), 0)
        return acc

    def step(self):
        p, s, h = self.p, self.s, 0.5 * self.p.dt
        moves = {"V": "F", "VL": "FL", "v": "f", "Hd": "H"}
        for m, a in self.acc.items():
            s[m] = s[m] + h * a
            if m in moves:
                s[moves[m]] = s[moves[m]] + p.dt * s[m]
            else:
                t, g = ("th", p.g_gauge) if m == "E" else ("th2", p.g_gauge2)
                v = s[t] - g * p.dx * p.dt * s[m]
                s[t] = v - 2 * math.pi * torch.round(v / (2 * math.pi))
        self.acc = self.force()
        for m, a in self.acc.items():
            s[m] = s[m] + h * a
            if self.damp is not None and m in ("V", "VL", "v", "E"):
                s[m] = s[m] * self.damp

    # -------------------------------------------------------- diagnostics

    def energies(self, F, V):
        p = self.p
        dV = p.dx ** 3
        Tp, Tm = transports(F, self.links() if p.gauged else None)
        D = [(a - b) / (2 * p.dx) for a, b in zip(Tp, Tm)]
        s = F[:3].abs().square()
        prod = s[0] * s[1] * s[2]
        sq = lambda z: float(z.abs().square().sum()) * dV  # noqa: E731
        cT = curl(D, 3)
        return dict(E_phi_kin=0.5 * sq(V[:3]), E_theta_kin=0.5 * sq(V[3:]), E_grad=0.5 * sum(sq(d[:3]) for d in D),
                    E_mass=0.5 * p.m2 * sq(F[:3]), E_pot=float((0.5 * p.mu * prod / (1 + p.kappa * prod)).sum()) * dV,
                    E_tgrad=0.5 * sum(sq(d[3:]) for d in D), E_tmass=0.5 * p.mtheta2 * sq(F[3:]),
                    E_coupling=-p.eta * dV * float((F[:3].real * cT.real + F[:3].imag * cT.imag).sum()))

    def real_row(self):
        p, f, v = self.p, self.s["f"], self.s["v"]
        dV, phi, th = p.dx ** 3, f[:3], f[3:]
        D = self.grads(f)
        cp, ct = curl(D, 0), curl(D, 3)
        sig, P = phi.square().sum(0), phi[0] * phi[1] * phi[2]
        m2 = p.inv_alpha / (1 + p.inv_beta * sig) if p.mode == 1 else p.m2
        pot = 0.5 * p.mu * P * P / (1 + p.kappa * P * P)
        if p.mode == 3:
            pot = 0.5 * p.mu * P * P * (1 + p.kappa_gamma * sig) / (1 + p.kappa_gamma * sig + p.kappa * P * P)
        pot = pot + p.alpha_cs * (0.5 * cp - th).square().sum(0) + p.kappa_h * P * P * (phi * cp).sum(0) + \
            0.5 * p.beta_h * th.square().sum(0) * cp.square().sum(0)
        tot = lambda z: float(z.sum()) * dV  # noqa: E731
        row = dict(E_phi_kin=0.5 * tot(v[:3].square()), E_theta_kin=0.5 * tot(v[3:].square()),
                   E_grad=0.5 * sum(tot(d[:3].square()) for d in D), E_mass=0.5 * tot(m2 * phi.square()),
                   E_pot=tot(pot), E_tgrad=0.5 * sum(tot(d[3:].square()) for d in D),
                   E_tmass=0.5 * p.mtheta2 * tot(th.square()), E_coupling=-p.eta * tot(phi * ct))
        row.update(E_total=sum(row.values()))
        row.update(phi_max=float(phi.abs().max()), P_max=float(P.abs().max()), P_int=tot(P.abs()),
                   theta_rms=math.sqrt(float(th.square().sum()) / (3 * p.N ** 3)))
        return row

    def row(self):
        p, s = self.p, self.s
        if p.real_fields:
            return self.vector(self.real_row())
        F, V, dV = s["F"], s["V"], p.dx ** 3
        X, Y, Z = axes(p)
        r2 = X * X + Y * Y + Z * Z
        row = self.energies(F, V)
        if "FL" in s:
            for k, v in self.energies(s["FL"], s["VL"]).items():
                row[k] += v
        sq = F[:3].abs().square()
        prod = sq[0] * sq[1] * sq[2]
        per = im_prod(F, V)
        Q = [float(per[a].sum()) * dV for a in range(6)]
        rho2 = sq.sum(0)
        m0 = float(rho2.sum())
        cen = [float((c * rho2).sum()) / m0 for c in (X, Y, Z)]
        spread = ((X - cen[0]) ** 2 + (Y - cen[1]) ** 2 + (Z - cen[2]) ** 2) * rho2
        at = int(torch.nonzero(prod.reshape(-1) >= prod.max() * (1 - 1e-12))[0])
        u, ud = F[0].reshape(-1)[at], V[0].reshape(-1)[at]
        place = lambda x: min(max(int(math.floor((x + p.L) / p.dx + 0.5)), 0), p.N - 1)  # noqa: E731
        c, i1, i2 = place(0.0), place(p.qdiag_probe1), place(p.qdiag_probe2)
        t1, t2 = complex(F[4, i1, c, c]), complex(F[4, i2, c, c])
        row.update(phi_max=float(sq.max().sqrt()), P_max=float(prod.max().sqrt()), P_int=float(prod.sqrt().sum()) * dV,
                   theta_rms=math.sqrt(float(F[3:].abs().square().sum()) / (6 * p.N ** 3)), Q_phi=sum(Q[:3]),
                   Q_theta=sum(Q[3:]), Q_total=sum(Q), s_max=float(prod.max()),
                   r_core=math.sqrt(float(spread.sum()) / m0),
                   omega_core=float(im_prod(u, ud)) / max(float(u.abs()) ** 2, 1e-300),
                   Q_core=float(per.sum(0)[r2 <= p.qdiag_radius ** 2].sum()) * dV, thp1u=t1.real, thp1v=t1.imag,
                   thp2u=t2.real, thp2v=t2.imag, Q_p0=Q[0], Q_p1=Q[1], Q_p2=Q[2], centroid_x=cen[0],
                   centroid_y=cen[1], centroid_z=cen[2])
        row["E_total"] = sum(row[k] for k in DIAG_NAMES[:8])
        if p.complex_gauge:
            dE = div(s["E"], p.dx)
            G = dE - p.g_gauge * self.rho_em() - self.offset
            inner = p.L - p.damp_width - p.dx if p.bc_type == 0 else 1e300
            G = G[(r2 < inner * inner).expand_as(G)]
            em = 0.5 * float(s["E"].square().sum()) + \
                float(sum((1 - c).sum() for c in plaquettes(s["th"], torch.cos))) / (p.g_gauge ** 2 * p.dx ** 4)
            R = p.qdiag_radius
            cube = ((X.abs() <= R) & (Y.abs() <= R) & (Z.abs() <= R))
            row.update(gauss_max=float(G.abs().max()), gauss_l2=math.sqrt(float(G.square().mean())), E_em=em * dV,
                       Q_flux=float((dE[cube] - self.offset).sum()) * dV / p.g_gauge)
            row["E_total"] += em * dV
        if "H" in s:
            H = s["H"]
            dens = 0.5 * s["Hd"].square() + 0.5 * sum(g.square() for g in self.grads(H)) + \
                0.25 * p.higgs_lam * (H * H - p.higgs_v ** 2).square() + 0.5 * p.higgs_kap * prod * H * H
            row["E_total"] += float(dens.sum()) * dV
        if "FL" in s:
            qc, ql = sum(Q), float(rho_of(s["FL"], s["VL"]).sum()) * dV
            row.update(Q_C=qc, Q_Q=qc, Q_L=ql, Q_em=(p.q_C + p.q_Q) * qc + p.q_L * ql)
        return self.vector(row)

    @staticmethod
    def vector(row):
        return np.array([row.get(k, 0.0) for k in DIAG_NAMES])

    def frame(self):
        return [c.reshape(-1).cpu().numpy() for c in columns(self.p, self.s)]


def exact(case, seed):
    if not torch.cuda.is_available() and case["n"] ** 3 * max(case["steps"], 1) > 1e7:
        return None   # minutes on host cores
    m = Plain(params_of(case), inputs(case, seed))
    if case["kind"] == "start":
        return dict(rows=np.stack([m.row()]), frame=m.frame())
    rows = []
    for n in range(1, case["steps"] + 1):
        m.step()
        if n % case["every"] == 0:
            rows.append(m.row())
    return dict(rows=np.stack(rows), frame=m.frame())
