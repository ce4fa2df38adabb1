"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is one call sequence through the public interface (mcf_gb300.SDPD) on one fluid: velocity-Verlet steps
of a resident state (run_vv), steps on the caller's own host arrays (step_vv_host), the right-hand side stage by stage as
MCF's driver calls it, or the stress adjoint.  Fluids, cut-offs and time steps are those of mcf_gb300/configs.py, in
boxes of nx x ny (x nz) lattice sites; the particles are disordered by a seeded jitter, as in a developed flow.

exact() integrates the same equations with plain torch in 64 bits: every pair found from explicit periodic or sheared ghost
copies, no part of the framework used.
"""
from __future__ import annotations

import math

import numpy as np
import torch

#: per fluid: lattice spacing, cut-off in spacings, sound speed, viscosity, kT, time step, body force (type, g_x)
FLUIDS = {
    "reverse": dict(dx=1.0 / 64, rc=3, c=10.0, eta=1.0, kt=0.0, dt=5e-5, body=(2, 1.0)),   # reverse Poiseuille
    "thermal": dict(dx=1.0, rc=3, c=10.0, eta=1.0, kt=1e-3, dt=1e-4, body=(0, 0.0)),       # fluctuating periodic box
    "channel": dict(dx=1.0, rc=3, c=20.0, eta=0.5, kt=1e-4, dt=5e-5, body=(1, 0.1)),       # Poiseuille between y walls
    "shear": dict(dx=1.0, rc=3, c=10.0, eta=1.0, kt=1e-4, dt=1e-3, body=(0, 0.0)),         # Lees-Edwards y faces
    "polymer": dict(dx=1.0, rc=3, c=10.0, eta=0.5, kt=1e-4, dt=1e-3, body=(3, 0.01)),      # Oldroyd-B
    "deck": dict(dx=0.1, rc=4, c=84.6, eta=8.46, kt=0.0, dt=2.6e-4, body=(0, 0.0)),        # MCF's scalability physics
    "colloids": dict(dx=1.0, rc=3, c=10.0, eta=1.0, kt=1e-3, dt=5e-5, body=(1, 0.05)),     # rigid spheres in solvent
}
WALL_LAYERS = 4        # ceil(1.05 rc / dx) for rc = 3 dx
SHEAR_RATE = 0.05
G, TAU = 0.5, 1.0      # polymer modulus n_p kT_p and relaxation time
RADIUS, HN = 4.0, 0.4  # colloid radius, range of their repulsion
WEIGHTS = (0.0, 1.0, 1.0)  # the adjoint's stress functional: off-diagonal entries


def listed():
    def case(name, work, fluid, size, steps, fp32, reuse):
        return dict(name=name, work=work, fluid=fluid, dim=len(size), nx=size[0], ny=size[1],
                    nz=size[2] if len(size) == 3 else 1, steps=steps, fp32=fp32, reuse=reuse)

    return [
        # a small 2D validation run in FP64, MCF's cell list rebuilt every step (the default): latency and launches
        case("2d_fp64_small", "run", "reverse", (64, 64), 20, False, False),
        # a 2D viscoelastic flow of the size that studies use, FP32-mixed
        case("2d_polymer", "run", "polymer", (128, 128), 20, True, True),
        # a small 3D channel, ragged in every direction, FP32-mixed
        case("3d_channel_small", "run", "channel", (33, 32, 31), 20, True, True),
        # the 1M-particle channel that production runs step through, FP32-mixed with the candidate list kept
        case("3d_channel_1m", "run", "channel", (100, 100, 100), 20, True, True),
        # the same precision with MCF's list rebuilt every step, uneven box
        case("3d_thermal_rebuild", "run", "thermal", (61, 64, 67), 10, True, False),
        # fluctuating hydrodynamics in FP64, the candidate list kept
        case("3d_thermal_fp64", "run", "thermal", (64, 64, 64), 5, False, True),
        # one right-hand side of an FP64 channel, stage by stage as MCF's driver calls it (slabs and parity work step so)
        case("3d_rhs_fp64", "rhs", "channel", (40, 41, 43), 1, False, False),
        # simple shear through Lees-Edwards faces
        case("3d_shear", "run", "shear", (80, 80, 80), 10, True, True),
        # MCF's own scalability deck: wide support, no noise, angular force
        case("3d_deck", "run", "deck", (80, 80, 80), 10, True, True),
        # a suspension of moving rigid spheres (their places depend on the box alone, so that every seed has the same particles)
        case("3d_colloids", "run", "colloids", (64, 64, 64), 10, True, True),
        # MCF's driver keeps x and v and hands them over each step
        case("3d_host_step", "host", "channel", (64, 64, 64), 8, True, True),
        # gradient of the mean stress by the adjoint (forward and backward)
        case("2d_adjoint", "adjoint", "polymer", (96, 96), 20, False, False),
    ]


def draw(rng):
    """Another fluid, call, size and precision of the same ranges; sizes spread over their logarithm."""
    work = rng.choice(["run"] * 7 + ["host", "rhs", "adjoint"])
    if work == "adjoint":
        fluid, fp32, reuse = rng.choice(["polymer", "thermal"]), False, False
        dim = 2 if fluid == "polymer" else 3
        n, steps = _log(rng, *((2500, 16000) if dim == 2 else (4000, 20000))), rng.randint(8, 20)
    elif work == "rhs":
        fluid, fp32, reuse = rng.choice(["reverse", "thermal", "channel"]), False, False
        dim = rng.choice([2, 3])
        n, steps = _log(rng, 4000, 200000), 1
    else:
        fluid = rng.choice(list(FLUIDS) if work == "run" else ["channel", "thermal"])
        dim = {"reverse": 2, "polymer": 2, "thermal": 3, "deck": 3, "colloids": 3}.get(fluid) or rng.choice([2, 3, 3])
        fp32 = rng.random() < 0.65
        reuse = work == "host" or rng.random() < (0.8 if fp32 else 0.5)
        n = _log(rng, 4000, 700000 if fp32 and fluid != "deck" else 260000 if fp32 else 200000)
        if fluid == "colloids":
            n = max(n, 40 ** 3)
        steps = rng.randint(5, 20) if n < 100000 else 5
    side = n ** (1.0 / dim)
    low = 36 if fluid == "colloids" else 14
    size = [max(low, int(round(side * rng.uniform(0.85, 1.15)))) for _ in range(dim)]
    return dict(work=work, fluid=fluid, dim=dim, nx=size[0], ny=size[1], nz=size[2] if dim == 3 else 1, steps=steps,
                fp32=fp32, reuse=reuse)


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


# ---------------------------------------------------------------- inputs
def _sites(case):
    return [case["nx"], case["ny"], case["nz"]][:case["dim"]]


def _fluid(case):
    f = FLUIDS[case["fluid"]]
    low = [0.0] * 3
    high = [n * f["dx"] for n in _sites(case)] + [0.0] * (3 - case["dim"])
    pad = WALL_LAYERS * f["dx"] if case["fluid"] == "channel" else 0.0
    return f, low, high, pad


def _particles(case, seed):
    """Positions, velocities, masses, ids (pid, sid), conformation tensor or None, colloids (centres, V, omega) or None."""
    f, low, high, pad = _fluid(case)
    dim, dx = case["dim"], f["dx"]
    rng = np.random.default_rng([int(seed), 77])
    axes = [(np.arange(n) + 0.5) * dx for n in _sites(case)]
    if pad:
        axes[1] = (np.arange(case["ny"] + 2 * WALL_LAYERS) + 0.5) * dx - pad
    x = np.stack([g.ravel() for g in np.meshgrid(*axes[::-1], indexing="ij")][::-1], axis=1)
    sid = np.zeros(len(x), np.int32)
    colloids = None
    if pad:
        sid[x[:, 1] < 0.0] = -3
        sid[x[:, 1] > high[1]] = -4
    if case["fluid"] == "colloids":
        box = np.array(high)
        centres = []
        for trial in np.random.default_rng(_sites(case)).uniform(0.0, 1.0, (4000, 3)) * box:
            d = np.array(centres).reshape(-1, 3) - trial
            d -= box * np.round(d / box)
            if len(centres) < len(x) // 4400 and (np.sqrt((d * d).sum(1)) > 2 * RADIUS + 1.0).all():
                centres.append(trial)
        centres = np.array(centres)
        keep = np.ones(len(x), bool)
        for k, c in enumerate(centres):
            d = x - c
            d -= box * np.round(d / box)
            r = np.sqrt((d * d).sum(1))
            sid[r <= RADIUS] = k + 1
            keep[r <= RADIUS - 1.05 * f["rc"] * dx] = False
        x, sid = x[keep], sid[keep]
        colloids = (centres, rng.normal(0.0, 0.02, centres.shape), rng.normal(0.0, 0.01, centres.shape))
    fluid = sid == 0
    x[fluid] += rng.uniform(-0.05 * dx, 0.05 * dx, (int(fluid.sum()), dim))
    v = np.zeros_like(x)
    v[fluid] = rng.normal(0.0, max(math.sqrt(f["kt"]), 1e-2 * dx), (int(fluid.sum()), dim))
    if case["fluid"] == "shear":
        v[:, 0] += SHEAR_RATE * (x[:, 1] - 0.5 * high[1])
    ct = None
    if case["fluid"] == "polymer":
        a = rng.normal(0.0, 0.05, (len(x), dim, dim))
        ct = (np.eye(dim) + a + a.transpose(0, 2, 1)).reshape(len(x), dim * dim)
    ids = np.stack([np.arange(1, len(x) + 1), sid], axis=1).astype(np.int32)
    return x, v, np.full(len(x), dx ** dim), ids, ct, colloids


def _params(case, seed):
    from mcf_gb300 import params as P
    f, low, high, pad = _fluid(case)
    bc, wall_v, low_t, high_t = [P.BC_PERIODIC] * 6, [[0.0] * 3 for _ in range(6)], list(low), list(high)
    if pad:
        bc[2] = bc[3] = P.BC_WALL_SOLID
        low_t[1], high_t[1] = -pad, high[1] + pad
    if case["fluid"] == "shear":
        bc[2] = bc[3] = P.BC_LE
        wall_v[2][0], wall_v[3][0] = -0.5 * SHEAR_RATE * high[1], 0.5 * SHEAR_RATE * high[1]
    p = P.make_params(num_dim=case["dim"], bcdef=bc, min_phys=low, max_phys=high, min_phys_t=low_t, max_phys_t=high_t,
                      cut_off=f["rc"] * f["dx"], c=f["c"], eta=f["eta"], kt=f["kt"], Brownian=1 if f["kt"] > 0 else 0, dt=f["dt"],
                      body_force_type=f["body"][0], body_force=[f["body"][1], 0.0, 0.0], wall_v=wall_v, seed=int(seed),
                      precision=P.PRECISION_FP32_MIXED if case["fp32"] else P.PRECISION_FP64)
    if case["fluid"] == "deck":
        for key, value in dict(rhs_force_type=4, eta_coef=4.0, stateEquation_type=2, rho_ref=0.9, gamma=7.0).items():
            setattr(p, key, value)
    if case["fluid"] == "polymer":
        for key, value in dict(Newtonian=0, tau=TAU, n_p=1.0, kt_p=G).items():
            setattr(p, key, value)
    p.stress_tensor = 1 if case["work"] == "adjoint" else 0
    p.reserved[1] = 1 if case["reuse"] else 0
    return p


def prepare(case, seed):
    from mcf_gb300.mcfg import SDPD
    from mcf_gb300.params import ColloidDynamics, ColloidParams
    x, v, m, ids, ct, colloids = _particles(case, seed)
    sim = SDPD(_params(case, seed))
    sim.upload(x, v, m, ids, ct)
    state = dict(case=case, sim=sim, step=0, dt=FLUIDS[case["fluid"]]["dt"])
    if case["work"] in ("rhs", "adjoint"):
        return dict(state, x=x, v=v, m=m, ids=ids, ct=ct)
    if colloids is not None:
        n = len(colloids[0])
        cp = ColloidParams(num_colloid=n, noslip_type=2, translate=1, rotate=1, cc_repul_type=2, dout=0.05, cc_repul_F0=10.0,
                           cc_repul_cut_off=HN, cc_repul_cut_on=0.1 * HN)
        sim.set_colloids(cp, *colloids, np.full(n, RADIUS))
        mass = np.full(n, 4.0 / 3.0 * math.pi * RADIUS ** 3)
        sim.set_colloid_dynamics(ColloidDynamics(integrate_AB=2, sub_time_step=1), mass,
                                 np.repeat(0.4 * mass[:, None] * RADIUS ** 2, 3, axis=1))
    sim.marching_init_force(0)
    if case["work"] == "host":
        sim.host_register(x)
        sim.host_register(v)
        state.update(x=x, v=v, pinned=_Pinned(sim, (x, v)))
    return state


class _Pinned:
    """Gives page-locked arrays back with the state that holds them."""

    def __init__(self, sim, arrays):
        self.sim, self.arrays = sim, arrays

    def __del__(self):
        for a in self.arrays:
            self.sim.host_unregister(a)


# ---------------------------------------------------------------- one pass
def run(state):
    case, sim, dt = state["case"], state["sim"], state["dt"]
    if case["work"] == "rhs":
        # MCF's driver, stage by stage on the arrays that it keeps
        sim.update_state(x=state["x"], v=state["v"])
        sim.technique_build_list(False)
        sim.particles_compute_density()
        sim.particles_compute_pressure()
        sim.particles_compute_interaction(1)
        sim.particles_apply_body_force()
        return sim.download("rho", "p", "f")
    if case["work"] == "adjoint":
        sim.upload(state["x"], state["v"], state["m"], state["ids"], state["ct"])
        d = case["dim"]
        w = np.array([[WEIGHTS[abs(a - b)] for b in range(d)] for a in range(d)])
        J, dp, grads = sim.adjoint_run(0, case["steps"], dt, w, checkpoint_every=10, state_grads=True)
        return dict(J=J, params=dp, **grads)
    first, state["step"] = state["step"], state["step"] + case["steps"]
    if case["work"] == "host":
        for k in range(case["steps"]):
            sim.step_vv_host(first + k + 1, dt, state["x"], state["v"])
        out = dict(x=state["x"].copy(), v=state["v"].copy())
    else:
        sim.run_vv(first, case["steps"], dt)
        # the computed columns of MCF's particle and restart files
        out = sim.download("x", "v", "rho", *(["ct"] if case["fluid"] == "polymer" else []))
    if case["fluid"] == "colloids":
        c = sim.colloid_state()
        out.update(centre=c["x"], V=c["v"][0], omega=c["omega"][0])
    if case["fp32"]:
        # positions are FP64 in both precisions; what the FP32 pair sums feed is kept in single precision
        out = {k: a if k in ("x", "centre") else torch.from_numpy(a).float() for k, a in out.items()}
    return out


def work(case):
    """Each step reads and writes x, v, f and reads mass and ids once; each pair is evaluated once: W and its sum about 25 flops,
    the force 75 (its random term 40 more, the conformation terms 30), the adjoint three times that again."""
    f, _, _, pad = _fluid(case)
    n = 1
    for s, a in zip(_sites(case), "xyz"):
        n *= s + (2 * WALL_LAYERS if pad and a == "y" else 0)
    d = case["dim"]
    pairs = 0.5 * n * (math.pi * f["rc"] ** 2 if d == 2 else 4.0 / 3.0 * math.pi * f["rc"] ** 3)
    flops = 100 + (40 if f["kt"] > 0 else 0) + (30 if case["fluid"] == "polymer" else 0)
    steps = case["steps"] * (4 if case["work"] == "adjoint" else 1)
    real = 6 * d * 8 + 16 + (2 * d * d * 8 if case["fluid"] == "polymer" else 0)
    return {"bytes": float(steps * n * real), "flops": float(steps * pairs * flops)}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, m, ids, ct, colloids = _particles(case, seed)
    ref = _Reference(case, seed, dev, m, ids, colloids)
    t = lambda a: None if a is None else torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    x, v, ct = t(x), t(v), t(ct)
    if case["work"] == "adjoint":
        return ref.gradients(x, v, ct)
    if case["work"] == "rhs":
        out = ref.rhs(x, v, ct, 1, 0.0)
        return dict(rho=out["rho"], p=out["p"], f=ref.with_body(x, out["f"]))
    out = ref.march(x, v, ct, case["steps"])
    names = ["x", "v"] if case["work"] == "host" else ["x", "v", "rho"]
    names += ["ct"] if ct is not None else []
    names += ["centre", "V", "omega"] if colloids is not None else []
    return {k: out[k] for k in names}


class _Reference:
    """Number-density SDPD in FP64 torch over explicit pairs and ghost copies."""

    def __init__(self, case, seed, dev, m, ids, colloids):
        self.case, self.dev, self.seed, self.dim = case, dev, int(seed), case["dim"]
        self.f, low, high, self.pad = _fluid(case)
        self.rc = self.f["rc"] * self.f["dx"]
        self.h = self.rc / 3.0
        self.m = float(m[0])
        self.box = torch.tensor(high[:self.dim], dtype=torch.float64, device=dev)
        self.pid = torch.tensor(ids[:, 0], dtype=torch.int64, device=dev)
        self.sid = torch.tensor(ids[:, 1], dtype=torch.int64, device=dev)
        self.colloids = None
        if colloids is not None:
            self.colloids = [torch.tensor(c, dtype=torch.float64, device=dev) for c in colloids]
        self.dv = SHEAR_RATE * high[1] if case["fluid"] == "shear" else 0.0
        self.eta, self.c, self.tau = self.f["eta"], self.f["c"], TAU

    # -- pairs
    def pairs(self, x, shift):
        """Ordered pairs (i, j) within the cut-off, the image's displacement and its x velocity; `shift`: of the sheared images."""
        n, d, rc = x.shape[0], self.dim, self.rc
        x = x.detach()
        src, pos, vel = torch.arange(n, device=self.dev), x, torch.zeros(n, dtype=x.dtype, device=self.dev)
        order = [1] + [a for a in range(d) if a != 1] if self.dv else range(d)
        for a in order:
            if self.pad and a == 1:
                continue
            more = [(src, pos, vel)]
            for sign in (1.0, -1.0):
                near = pos[:, a] < rc if sign > 0 else pos[:, a] >= self.box[a] - rc
                q = pos[near].clone()
                q[:, a] += sign * self.box[a]
                u = vel[near]
                if self.dv and a == 1:
                    q[:, 0] = torch.remainder(q[:, 0] + sign * shift, self.box[0])
                    u = u + sign * self.dv
                more.append((src[near], q, u))
            src, pos, vel = (torch.cat(t) for t in zip(*more))
        lo, hi = pos.min(0).values, pos.max(0).values
        nm = torch.clamp(((hi - lo) / rc).floor(), min=1).long()
        cell = torch.minimum(((pos - lo) / ((hi - lo) / nm)).floor().long(), nm - 1)
        row = cell[:, 1] if d == 2 else cell[:, 1] + nm[1] * cell[:, 2]
        key = row * nm[0] + cell[:, 0]
        by = torch.argsort(key)
        total = int(nm.prod())
        start = torch.zeros(total + 1, dtype=torch.int64, device=self.dev)
        start[1:] = torch.cumsum(torch.bincount(key, minlength=total), 0)
        got = []
        for c0 in range(0, n, 1 << 17):
            i = torch.arange(c0, min(n, c0 + (1 << 17)), device=self.dev)
            for oy in (-1, 0, 1):
                for oz in ((0,) if d == 2 else (-1, 0, 1)):
                    ry = cell[i, 1] + oy
                    rz = cell[i, 2] + oz if d == 3 else torch.zeros_like(ry)
                    ok = (ry >= 0) & (ry < nm[1]) & (rz >= 0) & ((rz < nm[2]) if d == 3 else True)
                    base = torch.where(ok, ry + (nm[1] * rz if d == 3 else 0), 0) * nm[0]
                    first = start[base + torch.clamp(cell[i, 0] - 1, min=0)]
                    count = torch.where(ok, start[base + torch.minimum(cell[i, 0] + 1, nm[0] - 1) + 1] - first, 0)
                    ii = torch.repeat_interleave(i, count)
                    within = torch.arange(ii.numel(), device=self.dev) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
                    g = by[torch.repeat_interleave(first, count) + within]
                    dist = ((x[ii] - pos[g]) ** 2).sum(1)
                    keep = (dist < rc * rc) & (g != ii)
                    got.append((ii[keep].int(), g[keep].int()))
        i, g = (torch.cat(t) for t in zip(*got))
        return i, g, src, pos - x[src], vel

    def sliced(self, pairs, x, v):
        """The pairs in pieces: i, j, separation, distance, and both velocities."""
        i, g, src, move, vel = pairs
        for k in range(0, i.numel(), 1 << 23):
            ii, gg = i[k:k + (1 << 23)].long(), g[k:k + (1 << 23)].long()
            j = src[gg]
            r = x[ii] - x[j] - move[gg]
            vj = v[j]
            if self.dv:
                vj = torch.cat([vj[:, :1] + vel[gg][:, None], vj[:, 1:]], 1)
            yield ii, j, r, (r * r).sum(1).sqrt(), v[ii], vj

    # -- kernel
    def coef(self):
        return 7.0 / (478.0 * math.pi * self.h ** 2) if self.dim == 2 else 3.0 / (359.0 * math.pi * self.h ** 3)

    def W(self, r):
        s = r / self.h
        p5 = lambda a: torch.clamp(a - s, min=0.0) ** 5  # noqa: E731
        return self.coef() * (p5(3.0) - 6.0 * p5(2.0) + 15.0 * p5(1.0))

    def dW(self, r):
        s = r / self.h
        p4 = lambda a: torch.clamp(a - s, min=0.0) ** 4  # noqa: E731
        return -5.0 * self.coef() / self.h * (p4(3.0) - 6.0 * p4(2.0) + 15.0 * p4(1.0))

    # -- random numbers: Philox4x32-10 keyed by the seed, counter (smaller pid, larger pid, step, 0), Box-Muller
    def normals(self, pa, pb, step):
        mask = 0xFFFFFFFF
        c = [torch.minimum(pa, pb), torch.maximum(pa, pb), torch.full_like(pa, step), torch.zeros_like(pa)]
        k0, k1 = self.seed & mask, (self.seed >> 32) & mask
        for _ in range(10):
            p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
            c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        u = [(2.0 * (w >> 9).double() + 1.0) * 2.0 ** -24 for w in c]
        out = []
        for a, b in ((u[0], u[1]), (u[2], u[3])):
            rad, angle = torch.sqrt(-2.0 * torch.log(a)), 2.0 * math.pi * b - math.pi
            out += [rad * torch.cos(angle), rad * torch.sin(angle)]
        return torch.stack(out[:self.dim], 1)

    # -- right-hand side
    def rhs(self, x, v, ct, step, shift):
        n, d, sid = x.shape[0], self.dim, self.sid
        pairs = self.pairs(x, shift)
        zero = torch.zeros(n, dtype=torch.float64, device=self.dev)
        rho = zero
        for i, j, r, dist, _, _ in self.sliced(pairs, x, v):
            rho = rho.index_add(0, i, self.W(dist))
        rho = torch.where(sid == 0, rho + 66.0 * self.coef(), 1.0 / self.m)
        dens = rho * self.m
        if self.case["fluid"] == "deck":
            p = self.c ** 2 * 0.9 ** 7.0 / 7.0 * ((dens / 0.9) ** 7.0 - 1.0)
        else:
            p = self.c ** 2 * (dens - 1.0)
        B = 1.0 / (rho * rho)
        c2 = None if ct is None else ct.reshape(n, d, d)
        f = torch.zeros_like(x)
        L = torch.zeros(n, d, d, dtype=torch.float64, device=self.dev)
        stress = torch.zeros_like(L[0])
        rx = self.relative(x) if self.colloids is not None else None
        for i, j, r, dist, vi, vj in self.sliced(pairs, x, v):
            si, sj = sid[i], sid[j]
            if self.pad or rx is not None:
                some = (si == 0) | (sj == 0)
                i, j, r, dist, vi, vj, si, sj = (t[some] for t in (i, j, r, dist, vi, vj, si, sj))
                vi, vj = self.no_slip(x, rx, i, j, r, vi, vj, si, sj)
            pi, pj = torch.where(si == 0, p[i], p[j]), torch.where(sj == 0, p[j], p[i])
            gw, e, vij = self.dW(dist), r / dist[:, None], vi - vj
            if self.case["fluid"] == "deck":
                a = (B[i] + B[j]) * gw
                g = ((4.0 * self.eta * a / dist * (e * vij).sum(1)) - a * 0.5 * (pi + pj))[:, None] * e
            else:
                extra = 0.0 if ct is None else G
                f_d = self.eta * (B[i] + B[j]) * gw / dist
                g = f_d[:, None] * vij - (((pi + extra) * B[i] + (pj + extra) * B[j]) * gw)[:, None] * e
                if self.f["kt"] > 0.0:
                    z = self.normals(self.pid[i], self.pid[j], step)
                    cb, ca = math.sqrt(0.5), math.sqrt(1.0 - 1.0 / d)
                    eg = (e * z).sum(1, keepdim=True)
                    amp = torch.sqrt(-4.0 * self.f["kt"] * f_d / self.f["dt"])
                    amp = torch.where(self.pid[i] < self.pid[j], amp, -amp)
                    g = g + amp[:, None] * (ca * eg * e + cb * (z - eg * e))
                if ct is not None:
                    Q = G * (c2[i] * B[i][:, None, None] + c2[j] * B[j][:, None, None])
                    g = g + (gw / dist)[:, None] * torch.einsum("pba,pa->pb", Q, r)
                    L = L.index_add(0, i, torch.einsum("pa,pb->pab", vj - vi, r) * (gw / dist / rho[i])[:, None, None])
            g = g / self.m
            f = f.index_add(0, i, g)
            if self.case["work"] == "adjoint":
                stress = stress + 0.5 * torch.einsum("pa,pb->ab", r, g)
        out = dict(rho=rho, p=p, f=f, stress=stress)
        if ct is not None:
            # tensors are stored column-major; c is symmetric
            t = torch.einsum("naq,nbq->nab", c2, L) + torch.einsum("naq,nqb->nab", L, c2)
            eye = torch.eye(d, dtype=torch.float64, device=self.dev)
            out["act"] = (t - (c2 - eye) / self.tau).reshape(n, d * d)
        return out

    def no_slip(self, x, rx, i, j, r, vi, vj, si, sj):
        """Morris' extrapolated velocity of a wall (at rest) or sphere boundary particle, on either side of the pair."""
        def of(fluid, other, so, vf, r_fo):
            if self.pad:
                face = torch.where(so == -3, 0.0, float(self.box[1]))
                a, b = x[fluid, 1] - face, x[other, 1] - face
                ratio = torch.where(a * b < 0.0, torch.clamp(b.abs() / a.abs(), max=0.5), 0.0)
                return -ratio[:, None] * vf
            _, V, om = self.colloids
            k = so - 1
            xc = rx[other]
            xf = xc + r_fo
            d = xf.norm(dim=1)
            gap = d - RADIUS
            ratio = torch.clamp((RADIUS - (xc * xf).sum(1) / d) / gap, -0.5, 0.5)[:, None]
            surface = V[k] + torch.linalg.cross(om[k], RADIUS / d[:, None] * xf)
            rigid = V[k] + torch.linalg.cross(om[k], xc)
            return torch.where((d <= RADIUS)[:, None], rigid, surface - ratio * (vf - surface))

        vi, vj = vi.clone(), vj.clone()
        b, a = sj != 0, si != 0
        new_j = of(i[b], j[b], sj[b], vi[b], r[b])
        new_i = of(j[a], i[a], si[a], vj[a], -r[a])
        vj[b], vi[a] = new_j, new_i
        return vi, vj

    def with_body(self, x, f):
        kind, g = self.f["body"]
        if kind == 0:
            return f
        if kind == 1:
            push = torch.full_like(x[:, 0], g)
        elif kind == 2:
            push = g * torch.sign(0.5 * self.box[-1] - x[:, -1])
        else:
            push = g * torch.sin(2.0 * math.pi / self.box[1] * x[:, 1])
        push = torch.where(self.sid == 0, push, 0.0)
        return torch.cat([f[:, :1] + push[:, None], f[:, 1:]], 1)

    # -- rigid spheres
    def relative(self, x):
        """Boundary particles relative to the nearest image of their centre (zero for solvent)."""
        d = x - self.colloids[0][torch.clamp(self.sid - 1, min=0)]
        d = d - self.box * torch.round(d / self.box)
        return torch.where((self.sid > 0)[:, None], d, 0.0)

    def rigid_v(self, x, v):
        if self.colloids is None:
            return v
        _, V, om = self.colloids
        k = torch.clamp(self.sid - 1, min=0)
        return torch.where((self.sid > 0)[:, None], V[k] + torch.linalg.cross(om[k], self.relative(x)), v)

    def spheres(self, x, f, step, hist):
        """Adams-Bashforth step of the spheres (order 1, then 2); returns the particles with the boundary ones moved."""
        X, V, om = self.colloids
        dt, mass = self.f["dt"], 4.0 / 3.0 * math.pi * RADIUS ** 3
        rx = self.relative(x)
        k, on = torch.clamp(self.sid - 1, min=0), (self.sid > 0)[:, None]
        push = torch.where(on, f * self.m, 0.0)
        drag = torch.zeros_like(X).index_add(0, k, push)
        torque = torch.zeros_like(X).index_add(0, k, torch.linalg.cross(rx, push))

        def repulsion(centres):
            r = centres[:, None] - centres[None]
            r = r - self.box * torch.round(r / self.box)
            dist = r.norm(dim=2)
            gap = dist - 2 * RADIUS
            near = (gap < 5 * HN) & ~torch.eye(len(X), dtype=torch.bool, device=self.dev)
            e1, e5 = torch.exp(-torch.clamp(gap, min=0.1 * HN) / HN), math.exp(-5.0)
            F = 10.0 / HN * (e1 / (1.0 - e1) - e5 / (1.0 - e5))
            F = torch.where(near, F / torch.where(near, dist, 1.0), 0.0)
            return (F[:, :, None] * r).sum(1)

        if not hist:  # the initial accelerations
            hist.update(V=V, om=om, F=(drag + repulsion(X)) / mass, al=torque / (0.4 * mass * RADIUS ** 2))
            hist["F0"], hist["al0"] = hist["F"], hist["al"]
        ab = (lambda a, b: a * dt) if step == 1 else (lambda a, b: (3.0 * a - b) * dt / 2.0)
        axis = ab(om, hist["om"])
        phi = axis.norm(dim=1, keepdim=True)
        u = (axis / phi)[k]
        c, s = torch.cos(phi)[k], torch.sin(phi)[k]
        turned = rx * c + torch.linalg.cross(u, rx) * s + u * (u * rx).sum(1, keepdim=True) * (1.0 - c)
        new = X + ab(V, hist["V"])
        F, al = hist["F"], hist["al"]
        hist["V"], hist["om"] = V, om
        V, om = V + ab(F, hist["F0"]), om + ab(al, hist["al0"])
        hist["F0"], hist["al0"] = F, al
        hist["F"], hist["al"] = (drag + repulsion(new)) / mass, torque / (0.4 * mass * RADIUS ** 2)
        self.colloids = [torch.remainder(new, self.box), V, om]
        return torch.where(on, new[k] + turned, x)

    # -- time stepping
    def wrap(self, x, v, shift):
        q = x.detach()
        if self.dv:
            over = torch.floor(q[:, 1] / self.box[1])
            x = torch.stack([x[:, 0] - over * shift, *x.unbind(1)[1:]], 1)
            v = torch.cat([v[:, :1] - (over * self.dv)[:, None], v[:, 1:]], 1)
        for_axis = torch.ones(self.dim, dtype=torch.float64, device=self.dev)
        if self.pad:
            for_axis[1] = 0.0
        return x - torch.floor(x.detach() / self.box) * self.box * for_axis, v

    def march(self, x, v, ct, steps, each=None):
        dt = self.f["dt"]
        fluid = (self.sid == 0)[:, None]
        out = self.rhs(x, self.rigid_v(x, v), ct, 0, 0.0)
        f, act, hist = self.with_body(x, out["f"]), out.get("act"), {}
        for k in range(1, steps + 1):
            shift = self.dv * (k + 1) * dt
            if self.colloids is not None:
                x = self.spheres(x, f, k, hist)
            v = torch.where(fluid, v + 0.5 * dt * f, v)
            x = torch.where(fluid, x + dt * v, x)
            x, v = self.wrap(x, v, shift)
            if ct is not None:
                ct = ct + 0.5 * dt * act
            v = self.rigid_v(x, v)
            out = self.rhs(x, v, ct, k, shift)
            f, act = self.with_body(x, out["f"]), out.get("act")
            v = torch.where(fluid, v + 0.5 * dt * f, v)
            if ct is not None:
                ct = ct + 0.5 * dt * act
            if each is not None:
                each(out)
        state = dict(x=x, v=v, rho=out["rho"], ct=ct)
        if self.colloids is not None:
            state.update(zip(("centre", "V", "omega"), self.colloids))
        return state

    def gradients(self, x, v, ct):
        """The mean of w : S over the steps and its gradient, by autograd through the trajectory."""
        leaf = lambda t: t.clone().requires_grad_(True)  # noqa: E731
        x0, v0, c0 = leaf(x), leaf(v), None if ct is None else leaf(ct)
        knobs = [leaf(torch.tensor(a, dtype=torch.float64, device=self.dev)) for a in (self.eta, self.tau, self.c)]
        self.eta, self.tau, self.c = knobs
        d = self.dim
        w = torch.tensor([[WEIGHTS[abs(a - b)] for b in range(d)] for a in range(d)], dtype=torch.float64, device=self.dev)
        stress = []
        self.march(x0, v0, c0, self.case["steps"], lambda o: stress.append((w * o["stress"]).sum()))
        J = sum(stress) / len(stress)
        wanted = knobs + [x0, v0] + ([] if c0 is None else [c0])
        g = torch.autograd.grad(J, wanted, allow_unused=True)
        out = dict(J=float(J.detach()), params=torch.stack([torch.zeros_like(J) if t is None else t for t in g[:3]]), x=g[3], v=g[4])
        if c0 is not None:
            out["ct"] = g[5]
        return out
