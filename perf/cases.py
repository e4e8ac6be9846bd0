"""Performance cases: what users of this library have it compute.

A user writes a HyPar deck (or fills a ``gb_config``), creates a solver and advances
Runge-Kutta steps; beside that plain path stand HyPar's function-pointer surface (one
right-hand side of a device array), the batched ensemble and the adjoint gradient.  The
cases below take each of these through the public Python classes at the sizes of the
repository's own workloads and tests, with odd and ragged ones among them.  ``run`` is one
call as such a program makes it; ``exact`` restates the same mathematics in plain 64-bit
torch, with nothing from this package.
"""
import math

import numpy as np
import torch

from hypar_gb300 import _lib
from hypar_gb300.solver import Ensemble, Solver, rk_table

GAMMA = 1.4
EPS = 1e-6
G = 3  # ghost points
MODEL_ND = {"euler1d": 1, "euler2d": 2, "navierstokes3d": 3}
BC_TYPE = {"periodic": 1, "extrapolate": 2, "slip-wall": 4}
RK_STAGES = {"44": 4, "ssprk3": 3, "22": 2}
# rising thermal bubble in a neutral atmosphere (SI units, 1 km cube)
ATMOS = {"R": 287.058, "rho": 1.1612055171196529, "p": 100000.0, "g": 9.8}
VISC = {"tgv": (1600.0, 0.72, 0.1), "turbulence": (333.333333333333333, 0.72, 0.3)}  # Re, Pr, Mach


def case(name, kind, model, size, flow, steps, interp="components", upwind="roe", weights="js", scheme="weno5",
         rk="44", bc="periodic", tuned=False):
    c = {"name": name, "kind": kind, "model": model, "flow": flow, "steps": steps, "interp": interp, "upwind": upwind,
         "weights": weights, "scheme": scheme, "rk": rk, "bc": bc, "tuned": tuned}
    for k, n in zip(("nx", "ny", "nz"), size):
        c[k] = n
    return c


def listed():
    return [
        # the Sod tube of the 1-D configuration: a short line, launch and latency bound; a
        # run of thousands of steps on a tuned solver
        case("sod_1024", "solve", "euler1d", [1024], "tube", 20, rk="44", bc="extrapolate", tuned=True),
        # a long 1-D line with characteristic reconstruction (shock-entropy interaction), as a deck runs it
        case("shock_entropy_20001", "solve", "euler1d", [20001], "entropy", 5, interp="characteristic",
             upwind="llf-char", rk="ssprk3", bc="extrapolate"),
        # the 2-D configuration: isentropic vortex, characteristic WENO5 + Roe, tuned
        case("vortex_1024", "solve", "euler2d", [1024, 1024], "vortex", 1, interp="characteristic", rk="ssprk3",
             tuned=True),
        # four-state Riemann problem on an odd rectangle, open ends: shocks and contacts in two dimensions
        case("riemann_601x403", "solve", "euler2d", [601, 403], "riemann", 2, interp="characteristic",
             upwind="rf-char", rk="ssprk3", bc="extrapolate"),
        # HyPar's own time integrator calling the right-hand side through the function pointers
        case("rhs_call_517x389", "rhs", "euler2d", [517, 389], "vortex", 1, upwind="llf-char"),
        # the 3-D configuration: Taylor-Green vortex, component-wise WENO5 + Roe + viscous term, classical RK4
        case("tgv_256", "solve", "navierstokes3d", [256, 256, 256], "tgv", 1),
        # decaying turbulence with mapped weights at an odd size
        case("turbulence_97", "solve", "navierstokes3d", [97, 97, 97], "turbulence", 1, weights="mapped", rk="ssprk3"),
        # the same flow with the compact scheme (line solves)
        case("turbulence_crweno_64", "solve", "navierstokes3d", [64, 64, 64], "turbulence", 1, weights="mapped",
             scheme="crweno5"),
        # rising thermal bubble: gravity, Rusanov, Yamaleev-Carpenter weights, slip walls, SI units
        case("bubble_64", "solve", "navierstokes3d", [64, 64, 64], "bubble", 1, upwind="rusanov", weights="yc",
             bc="slip-wall"),
        # 3-D characteristic reconstruction, inviscid, on a ragged box
        case("char3d_75x66x58", "solve", "navierstokes3d", [75, 66, 58], "tgv-inviscid", 1, interp="characteristic",
             rk="ssprk3"),
        # many small vortices advanced together
        case("ensemble_48", "ensemble", "euler2d", [32, 256], "vortex", 5, interp="characteristic", rk="ssprk3",
             tuned=True),
        # gradient of the final-time density misfit with respect to the initial density
        case("adjoint_256", "adjoint", "euler2d", [256, 256], "vortex", 6, rk="44"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["1d", "2d", "2d", "3d", "3d", "crweno", "bubble", "rhs", "ensemble", "adjoint"])
    interp = rng.choice(["components", "characteristic"])
    upwind = rng.choice(["roe", "llf-char", "rf-char"])
    rk = rng.choice(["44", "ssprk3"])
    if kind == "1d":
        flow = rng.choice(["tube", "entropy"])
        c = case("", "solve", "euler1d", [log(300, 30000)], flow, rng.randint(4, 20), interp, upwind, rk=rk,
                 bc="extrapolate")
    elif kind == "2d":
        flow = rng.choice(["vortex", "vortex", "riemann"])
        c = case("", "solve", "euler2d", [log(120, 1024), log(120, 1024)], flow, rng.randint(1, 2), interp, upwind,
                 rk=rk, bc="extrapolate" if flow == "riemann" else "periodic")
    elif kind == "3d":
        flow = rng.choice(["tgv", "turbulence", "tgv-inviscid"])
        size = [log(48, 160)] * 3 if flow == "turbulence" else [log(48, 160) for _ in range(3)]
        c = case("", "solve", "navierstokes3d", size, flow, 1, "components" if flow != "tgv-inviscid" else interp,
                 "roe" if flow != "tgv-inviscid" else upwind, rng.choice(["js", "mapped", "borges", "yc"]), rk=rk)
    elif kind == "crweno":
        c = case("", "solve", "navierstokes3d", [log(32, 96)] * 3, "turbulence", 1, scheme="crweno5",
                 weights=rng.choice(["js", "mapped"]), rk=rk)
    elif kind == "bubble":
        c = case("", "solve", "navierstokes3d", [log(40, 96)] * 3, "bubble", 1, upwind="rusanov", weights="yc", rk=rk,
                 bc="slip-wall")
    elif kind == "rhs":
        c = case("", "rhs", "euler2d", [log(100, 1024), log(100, 1024)], "vortex", 1, interp, upwind)
    elif kind == "ensemble":
        c = case("", "ensemble", "euler2d", [rng.choice([32, 48, 64]), rng.choice([128, 192, 256])], "vortex",
                 rng.randint(2, 5), interp, rng.choice(["roe", "llf-char"]), rk="ssprk3")
    else:
        n = log(64, 256)
        c = case("", "adjoint", "euler2d", [n, n], "vortex", rng.randint(3, 6), rk=rk)
    del c["name"]
    return c


def size_of(c):
    return [c[k] for k in ("nx", "ny", "nz")[:MODEL_ND[c["model"]]]]


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def generator(seed):
    return np.random.default_rng([int(seed), 20261205])


# --------------------------------------------------------------------------- initial states


def conserved(rho, vel, p):
    e = p / (GAMMA - 1.0) + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [e], dim=-1)


def grid(n, length, closed=False):
    h = length / (n - 1 if closed else n)
    return torch.arange(n, dtype=torch.float64, device=device()) * h, h


def vortex_state(n, rng, b=None, centre=None):
    """Isentropic vortex on [0,10)^2; n = (nx, ny)."""
    (x, hx), (y, hy) = grid(n[0], 10.0), grid(n[1], 10.0)
    Y, X = torch.meshgrid(y, x, indexing="ij")
    b = float(rng.uniform(4.0, 5.5)) if b is None else b
    xc, yc = (float(v) for v in rng.uniform(4.0, 6.0, 2)) if centre is None else centre
    r2 = (X - xc) ** 2 + (Y - yc) ** 2
    rho = (1.0 - (GAMMA - 1.0) * b * b / (8.0 * GAMMA * math.pi ** 2) * torch.exp(1.0 - r2)) ** (1.0 / (GAMMA - 1.0))
    q = b / (2.0 * math.pi) * torch.exp(0.5 * (1.0 - r2))
    return conserved(rho, [0.5 - q * (Y - yc), q * (X - xc)], rho ** GAMMA), [hx, hy]


def initial(c, seed):
    """The state in HyPar's order ([nz,] [ny,] nx, nvars) on the device, and the spacings."""
    rng, size, flow = generator(seed), size_of(c), c["flow"]
    if flow == "tube":
        x, h = grid(size[0], 1.0, closed=True)
        x0, pr, rr = rng.uniform(0.4, 0.6), rng.uniform(0.08, 0.12), rng.uniform(0.1, 0.15)
        one = torch.ones_like(x)
        left = x < float(x0)
        return conserved(torch.where(left, one, one * float(rr)), [0.0 * x], torch.where(left, one, one * float(pr))), [h]
    if flow == "entropy":  # Shu-Osher: a Mach 3 shock running into density waves
        x, h = grid(size[0], 10.0, closed=True)
        a, ph = float(rng.uniform(0.15, 0.25)), float(rng.uniform(0.0, 2.0 * math.pi))
        left = x < 1.0
        rho = torch.where(left, torch.full_like(x, 3.857143), 1.0 + a * torch.sin(5.0 * x + ph))
        vel = torch.where(left, torch.full_like(x, 2.629369), torch.zeros_like(x))
        return conserved(rho, [vel], torch.where(left, torch.full_like(x, 10.33333), torch.ones_like(x))), [h]
    if flow == "vortex":
        return vortex_state(size, rng)
    if flow == "riemann":  # four constant states, interfaces through a shifted centre
        (x, hx), (y, hy) = grid(size[0], 1.0, closed=True), grid(size[1], 1.0, closed=True)
        Y, X = torch.meshgrid(y, x, indexing="ij")
        xc, yc = (float(v) for v in rng.uniform(0.45, 0.8, 2))
        q = torch.where(X >= xc, torch.where(Y >= yc, 0, 3), torch.where(Y >= yc, 1, 2))
        vals = [(1.5, 0.0, 0.0, 1.5), (0.5323, 1.206, 0.0, 0.3), (0.138, 1.206, 1.206, 0.029), (0.5323, 0.0, 1.206, 0.3)]
        t = torch.tensor(vals, dtype=torch.float64, device=X.device)[q]
        return conserved(t[..., 0], [t[..., 1], t[..., 2]], t[..., 3]), [hx, hy]
    L = 2.0 * math.pi
    if flow in ("tgv", "tgv-inviscid"):
        axes = [grid(n, L) for n in size]
        Z, Y, X = torch.meshgrid(axes[2][0], axes[1][0], axes[0][0], indexing="ij")
        M = 0.1 if flow == "tgv" else 0.4
        sx, sy, sz = (float(v) for v in rng.uniform(0.0, L, 3))
        X, Y, Z = X + sx, Y + sy, Z + sz
        p = 1.0 / GAMMA + M * M / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
        vel = [M * torch.sin(X) * torch.cos(Y) * torch.cos(Z), -M * torch.cos(X) * torch.sin(Y) * torch.cos(Z),
               torch.zeros_like(X)]
        return conserved(torch.ones_like(X), vel, p), [a[1] for a in axes]
    if flow == "turbulence":  # solenoidal random field, Passot-Pouquet spectrum peaked at k = 4, rms Mach 0.3
        n = size[0]
        gen = torch.Generator(device=device()).manual_seed(int(seed) % (1 << 62))
        k1 = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=device())
        kr = torch.fft.rfftfreq(n, 1.0 / n, dtype=torch.float64, device=device())
        KZ, KY, KX = torch.meshgrid(k1, k1, kr, indexing="ij")
        k2 = KX * KX + KY * KY + KZ * KZ
        ks = torch.sqrt(torch.where(k2 > 0, k2, torch.ones_like(k2)))
        amp = torch.where(k2 > 0, torch.sqrt((ks / 4.0) ** 4 * torch.exp(-2.0 * (ks / 4.0) ** 2)) / ks, 0.0 * ks)
        xi = [torch.complex(*(torch.randn(k2.shape, dtype=torch.float64, device=device(), generator=gen) * amp
                              for _ in range(2))) for _ in range(3)]
        div = (KX * xi[0] + KY * xi[1] + KZ * xi[2]) / (ks * ks)
        vel = [torch.fft.irfftn(a - div * k, s=(n, n, n)) for a, k in zip(xi, (KX, KY, KZ))]
        rms = math.sqrt(sum(float((v * v).mean()) for v in vel) / 3.0)
        vel = [v * (0.3 / rms) for v in vel]
        one = torch.ones_like(vel[0])
        return conserved(one, vel, one / GAMMA), [L / n] * 3
    # bubble
    axes = [grid(n, 1000.0, closed=True) for n in size]
    Z, Y, X = torch.meshgrid(axes[2][0], axes[1][0], axes[0][0], indexing="ij")
    R, rho0, p0, g = ATMOS["R"], ATMOS["rho"], ATMOS["p"], ATMOS["g"]
    Cp, T0 = GAMMA * R / (GAMMA - 1.0), p0 / (R * rho0)
    cx, cy, cz = float(rng.uniform(450, 550)), float(rng.uniform(240, 300)), float(rng.uniform(450, 550))
    r = torch.sqrt((X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2)
    theta = T0 + torch.where(r > 250.0, torch.zeros_like(r), 0.5 * (1.0 + torch.cos(math.pi * r / 250.0)))
    exner = 1.0 - g * Y / (Cp * T0)
    rho = p0 / (R * theta) * exner ** (1.0 / (GAMMA - 1.0))
    zero = torch.zeros_like(rho)
    return conserved(rho, [zero, zero, zero], rho * R * theta * exner), [a[1] for a in axes]


def time_step(u, h, cfl=0.5):
    nd = u.dim() - 1
    rho = u[..., 0]
    vel = [u[..., 1 + d] / rho for d in range(nd)]
    p = (GAMMA - 1.0) * (u[..., -1] - 0.5 * rho * sum(v * v for v in vel))
    a = torch.sqrt(GAMMA * p / rho)
    return cfl / max(float(((v.abs() + a) / hd).max()) for v, hd in zip(vel, h))


def gravity_field(c, h):
    """Hydrostatic density and pressure factors of a neutral atmosphere along y, at every
    point with ghosts (mirrored into the ghost layers of each face)."""
    R, rho0, p0, g = ATMOS["R"], ATMOS["rho"], ATMOS["p"], ATMOS["g"]
    Cp, T0 = GAMMA * R / (GAMMA - 1.0), p0 / (R * rho0)
    ny = c["ny"]
    j = np.arange(-G, ny + G)
    j = np.where(j < 0, -1 - j, np.where(j >= ny, 2 * ny - 1 - j, j))
    ex = 1.0 - g * (j * h[1]) / (Cp * T0)
    return ex ** (-1.0 / (GAMMA - 1.0)), ex ** (GAMMA / (GAMMA - 1.0))


# --------------------------------------------------------------------------- prepare / run


def config(c, size, dt):
    """The deck of a case as a gb_config: whole-face boundaries, HyPar's extents."""
    nd = len(size)
    cfg = _lib.GbConfig()
    cfg.model, cfg.ndims, cfg.nvars, cfg.ghosts = _lib.MODEL[c["model"]], nd, nd + 2, G
    for d in range(3):
        cfg.dim[d] = size[d] if d < nd else 1
    cfg.interp, cfg.upwind = _lib.INTERP[c["interp"]], _lib.UPWIND[c["upwind"]]
    cfg.gamma, cfg.weno_eps = GAMMA, EPS
    cfg.Re, cfg.Pr, cfg.Minf = VISC.get(c["flow"], (-1.0, 0.72, 1.0))
    cfg.weno_weights, cfg.hyp_scheme, cfg.par_scheme = _lib.WENO_WEIGHTS[c["weights"]], _lib.SCHEME[c["scheme"]], 4
    z = 0
    for d in range(nd):
        for face in (1, -1):
            lo, hi = [0] * 3, [1] * 3
            for e in range(nd):
                lo[e], hi[e] = 0, size[e]
            lo[d], hi[d] = (-G, 0) if face == 1 else (size[d], size[d] + G)
            for k, v in enumerate([BC_TYPE[c["bc"]], d, face] + lo + hi):
                cfg.zones[z][k] = v
            z += 1
    cfg.nzones = z
    ns, A, b, cc = rk_table(c["rk"])
    cfg.rk_nstages = ns
    for k in range(16):
        cfg.rk_A[k] = A[k]
    for k in range(4):
        cfg.rk_b[k], cfg.rk_c[k] = b[k], cc[k]
    cfg.dt, cfg.n_iter, cfg.file_op_iter, cfg.screen_op_iter = dt, c["steps"], c["steps"], c["steps"]
    if c["flow"] == "bubble":
        cfg.gravity[1], cfg.rho_ref, cfg.p_ref = ATMOS["g"], ATMOS["rho"], ATMOS["p"]
        cfg.R_gas, cfg.HB = ATMOS["R"], 2
    return cfg


def dxinv(size, h):
    return np.concatenate([np.full(n + 2 * G, 1.0 / hd) for n, hd in zip(size, h)])


def solution(solver, out):
    """The solver's solution copied into the caller's device array (interior points)."""
    _lib.check(_lib.lib().gb_solver_get_state(solver.handle, out.data_ptr(), _lib.LAYOUT_INTERIOR, _lib.MEM_DEVICE))
    return out


def interior(t):
    return t[tuple(slice(G, -G) for _ in range(t.dim() - 1))]


def ensemble_members(c, seed):
    """(size, b, centre) of 48 vortices, sizes seeded from {nx, nx+16, ..., ny}^2."""
    rng = generator(seed)
    sizes = np.random.default_rng(7).choice(np.arange(c["nx"], c["ny"] + 1, 16), 48)  # one mix of sizes
    return [(int(n), float(rng.uniform(1.0, 5.0)), tuple(float(v) for v in rng.uniform(3.0, 7.0, 2))) for n in sizes]


def ensemble_states(c, seed):
    states = [vortex_state([n, n], None, b, xy) for n, b, xy in ensemble_members(c, seed)]
    return states, min(time_step(u, h) for u, h in states)


def adjoint_problem(c, seed):
    """Initial guess (a shifted, weaker vortex) and target density, and the step."""
    rng = generator(seed)
    size = size_of(c)
    sx, sy = (float(v) for v in rng.uniform(-0.5, 0.5, 2))
    u, h = vortex_state(size, None, 4.0, (5.0 + sx, 5.0 + sy))
    target, _ = vortex_state(size, None, 5.0, (5.0, 5.0))
    return u, target[..., 0].contiguous(), h, time_step(target, h)


def prepare(c, seed):
    size = size_of(c)
    if c["kind"] == "ensemble":
        states, dt = ensemble_states(c, seed)
        e = Ensemble([config(c, [u.shape[1], u.shape[0]], dt) for u, _ in states],
                     [dxinv([u.shape[1], u.shape[0]], h) for u, h in states])
        for m, (u, _) in enumerate(states):
            e.set_state(m, u.reshape(-1).cpu().numpy())
        if c["tuned"]:
            e.autotune(1)
        return {"case": c, "ensemble": e}
    if c["kind"] == "adjoint":
        from hypar_gb300.adjoint import Adjoint
        u, target, h, dt = adjoint_problem(c, seed)
        return {"case": c, "adjoint": Adjoint(config(c, size, dt), dxinv(size, h), c["steps"]), "u": u, "target": target}
    u, h = initial(c, seed)
    s = Solver(config(c, size, time_step(u, h)), dxinv(size, h))
    if c["flow"] == "bubble":
        f, g = (np.broadcast_to(v[None, :, None], [n + 2 * G for n in reversed(size)]).reshape(-1)
                for v in gravity_field(c, h))
        s.set_gravity_field(np.concatenate([f, g]))
    s.set_state(u.contiguous())
    if c["tuned"]:
        s.autotune(1)
    if c["kind"] == "rhs":
        ug = torch.zeros([n + 2 * G for n in reversed(size)] + [s.nvars], dtype=torch.float64, device=u.device)
        interior(ug).copy_(u)
        return {"case": c, "solver": s, "u": ug, "out": torch.empty_like(ug)}
    u = u.contiguous()
    return {"case": c, "solver": s, "u": u, "out": torch.empty_like(u)}


def run(state):
    c = state["case"]
    if c["kind"] == "ensemble":
        e = state["ensemble"]
        e.step(c["steps"])
        return [e.get_state(m) for m in range(len(e))]
    if c["kind"] == "adjoint":
        from hypar_gb300.adjoint import density_misfit_gradient
        loss, grad = density_misfit_gradient(state["adjoint"], state["u"], state["target"])
        return {"loss": loss, "gradient": grad}
    s = state["solver"]
    if c["kind"] == "rhs":
        s.rhs(state["out"], state["u"])
        return interior(state["out"])
    s.set_state(state["u"])
    s.step(c["steps"])
    return solution(s, state["out"])


def work(c):
    """Bytes: the state in and out once.  Flops: the scheme's arithmetic per cell, direction
    and stage (four biased WENO5 values of each component with their weights, the cell flux
    and the upwinding), plus the viscous term's."""
    nd = MODEL_ND[c["model"]]
    nv = nd + 2
    if c["kind"] == "ensemble":
        cells = sum(n * n for n, _, _ in ensemble_members(c, 0))
    else:
        cells = int(np.prod(size_of(c)))
    per = nv * (4 * 55 + 20) + 40 + (nv * nv * 24 if c["interp"] == "characteristic" else nv * nv * 4)
    if c["scheme"] == "crweno5":
        per += nv * 4 * 12
    evals = 1 if c["kind"] == "rhs" else c["steps"] * RK_STAGES[c["rk"]]
    flops = cells * evals * (per * nd + (600 if c["flow"] in VISC else 0))
    byts = 2 * 8 * nv * cells
    if c["kind"] == "adjoint":
        flops *= 3
        byts = 8 * cells * (nv + 2)
    return {"bytes": byts, "flops": flops}


# --------------------------------------------------------------------------- 64-bit restatement


def along(d):
    """Dimension d (0 fastest) of an array whose grid axes come last, slowest first."""
    return -1 - d


def pad(u, d, bc, normal=None):
    """Three ghost layers along d; `normal`: the component whose sign a slip wall flips."""
    ax = along(d)
    n = u.shape[ax]
    if bc == "periodic":
        return torch.cat([u.narrow(ax, n - G, G), u, u.narrow(ax, 0, G)], ax)
    lo, hi = u.narrow(ax, 0, G).flip(ax), u.narrow(ax, n - G, G).flip(ax)
    if bc == "slip-wall" and normal is not None:
        sign = torch.ones([u.shape[0]] + [1] * (u.dim() - 1), dtype=u.dtype, device=u.device)
        sign[normal] = -1.0
        lo, hi = lo * sign, hi * sign
    return torch.cat([lo, u, hi], ax)


def primitive(u):
    nd = u.shape[0] - 2
    rho = u[0]
    vel = [u[1 + d] / rho for d in range(nd)]
    return rho, vel, (GAMMA - 1.0) * (u[-1] - 0.5 * rho * sum(v * v for v in vel))


def flux_of(u, d):
    rho, vel, p = primitive(u)
    f = [rho * vel[d]] + [rho * v * vel[d] for v in vel] + [(u[-1] + p) * vel[d]]
    f[1 + d] = f[1 + d] + p
    return torch.stack(f)


def nonlinear_weights(m, opt, kind):
    b = [13.0 / 12.0 * (m[0] - 2 * m[1] + m[2]) ** 2 + 0.25 * (m[0] - 4 * m[1] + 3 * m[2]) ** 2,
         13.0 / 12.0 * (m[1] - 2 * m[2] + m[3]) ** 2 + 0.25 * (m[1] - m[3]) ** 2,
         13.0 / 12.0 * (m[2] - 2 * m[3] + m[4]) ** 2 + 0.25 * (3 * m[2] - 4 * m[3] + m[4]) ** 2]
    if kind in ("borges", "yc"):
        tau = (b[2] - b[0]).abs() if kind == "borges" else (m[0] - 4 * m[1] + 6 * m[2] - 4 * m[3] + m[4]) ** 2
        a = [o * (1.0 + (tau / (x + EPS)) ** 2) for o, x in zip(opt, b)]
    else:
        a = [o / (x + EPS) ** 2 for o, x in zip(opt, b)]
    s = a[0] + a[1] + a[2]
    w = [x / s for x in a]
    if kind == "mapped":
        a = [x * (o + o * o - 3 * o * x + x * x) / (o * o + x * (1.0 - 2.0 * o)) for o, x in zip(opt, w)]
        s = a[0] + a[1] + a[2]
        w = [x / s for x in a]
    return w


def candidates(m):
    return [(2 * m[0] - 7 * m[1] + 11 * m[2]) / 6, (-m[1] + 5 * m[2] + 2 * m[3]) / 6, (2 * m[2] + 5 * m[3] - m[4]) / 6]


WENO_OPT, CRWENO_OPT = (0.1, 0.6, 0.3), (0.2, 0.5, 0.3)


def weno5(m, values, kind):
    w = nonlinear_weights(m, WENO_OPT, kind)
    return sum(a * p for a, p in zip(w, candidates(values)))


def compact_weno5(sten, values, kind, ax, left):
    """CRWENO5 on every line along `ax`: explicit WENO5 rows at the two end interfaces, the
    compact rows between, one tridiagonal solve."""
    n = sten[0].shape[ax]
    w = nonlinear_weights(sten, CRWENO_OPT, kind)
    m = values
    rhs = (w[0] * (m[1] + 5 * m[2]) + w[1] * (5 * m[2] + m[3]) + w[2] * (m[2] + 5 * m[3])) / 6
    sub, dia, sup = (2 * w[0] + w[1]) / 3, (w[0] + 2 * w[1] + 2 * w[2]) / 3, w[2] / 3
    if not left:
        sub, sup = sup, sub
    explicit = weno5(sten, values, kind)
    a, b, s, r = (list(t.unbind(ax)) for t in (sub, dia, sup, rhs))
    e = explicit.unbind(ax)
    for i in (0, n - 1):
        a[i], b[i], s[i], r[i] = 0 * a[i], 0 * b[i] + 1, 0 * s[i], e[i]
    for i in range(1, n):
        k = a[i] / b[i - 1]
        b[i] = b[i] - k * s[i - 1]
        r[i] = r[i] - k * r[i - 1]
    for i in range(n - 1, -1, -1):
        r[i] = (r[i] - s[i] * r[i + 1]) / b[i] if i < n - 1 else r[i] / b[i]
    return torch.stack(r, ax)


def roe_average(a, b):
    """Velocity, enthalpy, density, sound speed of the Roe average of two conserved states."""
    (ra, va, pa), (rb, vb, pb) = primitive(a), primitive(b)
    ta, tb = torch.sqrt(ra), torch.sqrt(rb)
    s = ta + tb
    vel = [(ta * x + tb * y) / s for x, y in zip(va, vb)]
    H = (ta * (a[-1] + pa) / ra + tb * (b[-1] + pb) / rb) / s
    c = torch.sqrt((GAMMA - 1.0) * (H - 0.5 * sum(v * v for v in vel)))
    return vel, H, ta * tb, c


def project(avg, q, d):
    """Left eigenvectors of direction d applied to q: acoustic -, acoustic +, entropy, shears."""
    vel, _, rho, c = avg
    scale = 1.0 / (rho * c) if len(vel) == 1 else 0.5 / (c * c)
    s = (GAMMA - 1.0) * (0.5 * sum(v * v for v in vel) * q[0] - sum(v * m for v, m in zip(vel, q[1:])) + q[-1])
    t = c * (vel[d] * q[0] - q[1 + d])
    return torch.stack([(s + t) * scale, (s - t) * scale, q[0] - s / (c * c)]
                       + [v * q[0] - q[1 + e] for e, v in enumerate(vel) if e != d])


def unproject(avg, w, d):
    vel, H, rho, c = avg
    r = 0.5 * rho / c if len(vel) == 1 else 1.0
    wm, wp = w[0] * r, w[1] * r
    y0 = wm + wp + w[2]
    y = [y0] + [v * y0 for v in vel]
    y[1 + d] = y[1 + d] + c * (wp - wm)
    e = H * (wm + wp) + vel[d] * c * (wp - wm) + 0.5 * sum(v * v for v in vel) * w[2]
    k = 3
    for i, v in enumerate(vel):
        if i != d:
            y[1 + i] = y[1 + i] - w[k]
            e = e - v * w[k]
            k += 1
    return torch.stack(y + [e])


def eigenvalues(vel, c, d):
    return torch.stack([vel[d] - c, vel[d] + c] + [vel[d]] * len(vel))


def state_eigenvalues(u, d):
    rho, vel, p = primitive(u)
    return eigenvalues(vel, torch.sqrt(GAMMA * p / rho), d)


def numerical_flux(c, fL, fR, uL, uR, cl, cr, d, kappa):
    nd, up = cl.shape[0] - 2, c["upwind"]
    if up == "rusanov":
        def speed(vel, a):
            return a + vel[d].abs()
        (rl, vl, pl), (rr, vr, pr) = primitive(cl), primitive(cr)
        avg = roe_average(cl, cr)
        al = torch.maximum(torch.maximum(speed(vl, torch.sqrt(GAMMA * pl / rl)), speed(vr, torch.sqrt(GAMMA * pr / rr))),
                           speed(avg[0], avg[3]))
        return 0.5 * (fL + fR) - kappa * al * 0.5 * (uR - uL)
    own = nd == 2 or (nd == 3 and up != "roe")  # averages the reconstructed states
    avg = roe_average(uL, uR) if own else roe_average(cl, cr)
    lam = eigenvalues(avg[0], avg[3], d)
    if up == "roe":
        a = lam.abs()
        if nd > 1:
            a = torch.where(a < 1e-6, (lam * lam + 1e-12) / 2e-6, a)
        return 0.5 * (fL + fR) - unproject(avg, a * project(avg, 0.5 * (uR - uL), d), d)
    lL, lR = (state_eigenvalues(q, d) for q in ((cl, cr) if nd == 1 else (uL, uR)))
    fcL, fcR = project(avg, fL, d), project(avg, fR, d)
    al = torch.maximum(torch.maximum(lL.abs(), lam.abs()), lR.abs())
    fc = 0.5 * (fcL + fcR + al * project(avg, uL - uR, d))
    if up == "rf-char":
        fc = torch.where((lL > 0) & (lam > 0) & (lR > 0), fcL, torch.where((lL < 0) & (lam < 0) & (lR < 0), fcR, fc))
    return unproject(avg, fc, d)


def hyperbolic(c, u, h, grav):
    """-(sum over d of the flux differences), with the balanced source term under gravity."""
    nd = u.shape[0] - 2
    total = torch.zeros_like(u)
    for d in range(nd):
        ax = along(d)
        n = u.shape[ax]
        up = pad(u, d, c["bc"], 1 + d)
        f = flux_of(up, d)
        um = up
        kappa, S = 1.0, None
        if grav is not None:
            gf, gg = (pad(q.expand(u.shape[1:]), d, c["bc"]) for q in grav)
            rho, vel, p = primitive(up)
            um = torch.cat([up[:-1] * gf, (p / (GAMMA - 1.0) / gg + 0.5 * rho * sum(v * v for v in vel) * gf)[None]])
            kappa = torch.maximum(gg.narrow(ax, 2, n + 1), gg.narrow(ax, 3, n + 1))

        def win(q, k):
            return q.narrow(ax, k, n + 1)

        cl, cr = win(up, 2), win(up, 3)
        left, right = (0, 1, 2, 3, 4), (5, 4, 3, 2, 1)
        if c["interp"] == "characteristic":
            avg = roe_average(cl, cr)
            rec = []
            for w, v in ((f, f), (up, um)):
                pw = [project(avg, win(w, k), d) for k in range(6)]
                pv = pw if v is w else [project(avg, win(v, k), d) for k in range(6)]
                rec += [unproject(avg, weno5([pw[k] for k in s], [pv[k] for k in s], c["weights"]), d)
                        for s in (left, right)]
        else:
            rec = []
            for w, v in ((f, f), (up, um)):
                for s in (left, right):
                    rows = []
                    for q in range(u.shape[0]):  # one component at a time: less memory
                        sw, sv = [win(w[q], k) for k in s], [win(v[q], k) for k in s]
                        rows.append(compact_weno5(sw, sv, c["weights"], ax, s is left) if c["scheme"] == "crweno5"
                                    else weno5(sw, sv, c["weights"]))
                    rec.append(torch.stack(rows))
        F = numerical_flux(c, rec[0], rec[1], rec[2], rec[3], cl, cr, d, kappa)
        total = total - (F.narrow(ax, 1, n) - F.narrow(ax, 0, n)) / h[d]
        if grav is not None and d == 1:
            rho, vel, _ = primitive(u)
            term = rho * (ATMOS["p"] / ATMOS["rho"]) * gf.narrow(ax, G, n)
            for q, t in ((1 + d, term), (u.shape[0] - 1, term * vel[d])):
                sides = []
                for s in (left, right):
                    wts = nonlinear_weights([win(f[q], k) for k in s], WENO_OPT, c["weights"])
                    sides.append(sum(a * p for a, p in zip(wts, candidates([win(gg, k) for k in s]))))
                SI = 0.5 * (sides[0] + sides[1])
                total[q] = total[q] + t * (SI.narrow(ax, 1, n) - SI.narrow(ax, 0, n)) / h[d]
    return total


def derivative4(q, ax):
    """Fourth-order first difference along a ghost-extended line, one-sided at its ends."""
    n = q.shape[ax]

    def at(i):
        return q.narrow(ax, i, 1)

    mid = (q.narrow(ax, 0, n - 4) - 8 * q.narrow(ax, 1, n - 4) + 8 * q.narrow(ax, 3, n - 4) - q.narrow(ax, 4, n - 4)) / 12
    first = (-25 * at(0) + 48 * at(1) - 36 * at(2) + 16 * at(3) - 3 * at(4)) / 12
    second = (-3 * at(0) - 10 * at(1) + 18 * at(2) - 6 * at(3) + at(4)) / 12
    last = (25 * at(n - 1) - 48 * at(n - 2) + 36 * at(n - 3) - 16 * at(n - 4) + 3 * at(n - 5)) / 12
    before = (3 * at(n - 1) + 10 * at(n - 2) - 18 * at(n - 3) + 6 * at(n - 4) - at(n - 5)) / 12
    return torch.cat([first, second, mid, before, last], ax)


def viscous(c, u, h):
    """The fourth-order viscous term; across a ghost direction derivatives are zero at ghost points."""
    Re, Pr, Mach = VISC[c["flow"]]
    re = Re / Mach
    rho, vel, p = primitive(u)
    Q = torch.stack(vel + [GAMMA * p / rho])
    total = torch.zeros_like(u)
    D = [derivative4(pad(Q, e, "periodic"), along(e)) / h[e] for e in range(3)]
    inner = [q.narrow(along(e), G, q.shape[along(e)] - 2 * G) for e, q in enumerate(D)]
    for d in range(3):
        ax = along(d)
        Qg = pad(Q, d, "periodic")
        zero = torch.zeros_like(Q.narrow(ax, 0, G))
        g = [D[d] if e == d else torch.cat([zero, inner[e], zero], ax) for e in range(3)]
        mu = torch.exp(0.76 * torch.log(Qg[3])) / re
        div = g[0][0] + g[1][1] + g[2][2]
        tau = [mu * (g[e][d] + g[d][e]) if e != d else 2.0 / 3.0 * mu * (3 * g[d][d] - div) for e in range(3)]
        heat = mu / ((GAMMA - 1.0) * Pr) * g[d][3]
        F = torch.stack([torch.zeros_like(mu)] + tau + [sum(v * t for v, t in zip(Qg[:3], tau)) + heat])
        total = total + derivative4(F, ax).narrow(ax, G, u.shape[ax]) / h[d]
    return total


TABLES = {"44": ([[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6]),
          "ssprk3": ([[], [1.0], [0.25, 0.25]], [1 / 6, 1 / 6, 2 / 3])}


def advance(c, u, h, dt, steps, grav=None):
    A, b = TABLES[c["rk"]]

    def rhs(v):
        k = hyperbolic(c, v, h, grav)
        return k + viscous(c, v, h) if c["flow"] in VISC else k

    for _ in range(steps):
        ks = []
        for row in A:
            ks.append(rhs(u + dt * sum(a * k for a, k in zip(row, ks) if a) if ks else u))
        u = u + dt * sum(w * k for w, k in zip(b, ks))
    return u


def components_first(u):
    return u.movedim(-1, 0).contiguous()


def exact(c, seed):
    if c["kind"] == "ensemble":
        states, dt = ensemble_states(c, seed)
        return [advance(c, components_first(u), h, dt, c["steps"]).movedim(0, -1).reshape(-1).cpu().numpy()
                for u, h in states]
    if c["kind"] == "adjoint":
        u, target, h, dt = adjoint_problem(c, seed)
        u = components_first(u).requires_grad_(True)
        loss = 0.5 * ((advance(c, u, h, dt, c["steps"])[0] - target) ** 2).sum()
        loss.backward()
        return {"loss": float(loss.detach()), "gradient": u.grad[0]}
    u, h = initial(c, seed)
    if c["kind"] == "rhs":
        return hyperbolic(c, components_first(u), h, None).movedim(0, -1)
    grav = None
    if c["flow"] == "bubble":
        grav = [torch.tensor(v[G:-G], dtype=torch.float64, device=u.device)[None, :, None]
                for v in gravity_field(c, h)]
    return advance(c, components_first(u), h, time_step(u, h), c["steps"], grav).movedim(0, -1)
