"""Performance cases: what a program of this framework has it do, through `ziran2019_b200.mpm` and
`ziran2019_b200.rollout`.

A pass takes a simulation from a device checkpoint a number of substeps forward and reads the particles
back, as a program does once per output frame (`reverse` cases: a rollout and its gradients).  The scenes
are jittered blocks of `nx` x `ny` x `nz` cells with `ppc` particles each, in motion and deformed, against
colliders; materials, grid spacings, time steps and solver settings are those of `workloads.py`.

A case: `path` (integrator: newton, explicit, admm, reverse), `material`, `precision` (fp64, mixed),
`nx`, `ny`, `nz`, `ppc`, `steps` (substeps per pass), `mls` (explicit substeps: the MLS-MPM force).
"""
import math

import numpy as np
import torch

from ziran2019_b200 import abi, mpm, rollout

RHO = 1000.0

# grid spacing, log2 of the grid's extent, time step of an implicit substep, gravity, E, nu
SCENES = {
    "rubber": (1.0 / 64, 7, 1e-3, -9.8, 1e4, 0.3),     # fixed corotated, Newton-CG to 1e-7
    "elastic": (1.0 / 256, 9, 5e-4, -9.8, 5e4, 0.35),  # StVK-Hencky, Newton-MINRES (the library's defaults)
    "metal": (1.0 / 256, 9, 5e-4, -9.8, 5e4, 0.35),    # the same with von Mises plasticity
    "sand": (1.0 / 256, 9, 5e-4, -9.8, 5e4, 0.35),     # the same with Drucker-Prager plasticity
    "brittle": (1.0 / 216, 9, 2e-4, 0.0, 1e5, 0.3),    # neo-Hookean with Rankine damage, ends pulled apart
    "cracking": (1.0 / 216, 9, 2e-4, 0.0, 1e5, 0.3),   # neo-Hookean with the CD-MPM phase field, ends pulled apart
    "foam": (1.0 / 120, 8, 2e-3, -9.8, 2e4, 0.4),      # StVK-Hencky with a viscoelastic part, on a sphere
}
DT_EXPLICIT = 1e-4
YIELD = 150.0
FRICTION = 30.0
SIGMA_F, RESIDUAL = 1e3, 1e-3
REVERSE_SPREAD = 0.3


def listed():
    def case(name, path, material, precision, cells, steps, ppc=8, mls=False):
        return {"name": name, "path": path, "material": material, "precision": precision, "nx": cells[0], "ny": cells[1],
                "nz": cells[2], "ppc": ppc, "steps": steps, "mls": mls}
    return [
        # a small interactive scene: launch and host latency are what it feels
        case("rubber-4k-mixed", "newton", "rubber", "mixed", (8, 8, 8), 4),
        # a ragged coarse preview in the reference's double layout
        case("elastic-33k-fp64", "newton", "elastic", "fp64", (17, 13, 19), 10),
        # the benchmark's elastoplastic scene at full size
        case("metal-1m-mixed", "newton", "metal", "mixed", (50, 50, 50), 20),
        # the same scene's quarter, all in double
        case("metal-250k-fp64", "newton", "metal", "fp64", (25, 25, 50), 10),
        # a mid-size granular column of odd extents
        case("sand-197k-mixed", "newton", "sand", "mixed", (37, 29, 23), 10),
        # short explicit substeps of a large scene
        case("explicit-1m-mixed", "explicit", "metal", "mixed", (50, 50, 50), 40),
        # explicit MLS-MPM substeps of a small scene in double
        case("explicit-mls-60k-fp64", "explicit", "elastic", "fp64", (19, 23, 17), 20, mls=True),
        # the viscoelastic slab on a sphere at full size: 20 ADMM iterations a substep
        case("admm-498k-mixed", "admm", "foam", "mixed", (72, 12, 72), 2),
        # a cut of it in double
        case("admm-31k-fp64", "admm", "foam", "fp64", (18, 12, 18), 2),
        # a quarter of the notched slab's volume with Rankine damage, damage read back for output
        case("brittle-513k-mixed", "newton", "brittle", "mixed", (108, 54, 11), 10),
        # a phase-field fracture specimen in double, the phase field read back for output
        case("cracking-84k-fp64", "newton", "cracking", "fp64", (54, 27, 9), 10, ppc=6),
        # gradients of a short rollout with respect to stiffness and initial velocity
        case("reverse-64k-mixed", "reverse", "rubber", "mixed", (20, 20, 20), 4),
    ]


# most particles, and most particles x substeps of a pass, that a drawn case has (below the listed ones of its kind)
_LIMITS = {"newton": (1_000_000, 6_000_000), "explicit": (1_000_000, 30_000_000), "admm": (400_000, 600_000), "reverse": (60_000, 160_000)}


def draw(rng):
    path = rng.choice(["newton", "newton", "newton", "explicit", "explicit", "admm", "reverse"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    material = {"newton": lambda: rng.choice(["rubber", "elastic", "metal", "sand", "brittle", "cracking"]),
                "explicit": lambda: rng.choice(["elastic", "metal", "sand"]),
                "admm": lambda: "foam", "reverse": lambda: "rubber"}[path]()
    most, work = _LIMITS[path]
    if precision == "fp64":
        most, work = most // 2, work // 2
    if material == "cracking":
        most, work = most // 3, work // 3
    particles = math.exp(rng.uniform(math.log(3000), math.log(most)))
    ppc = rng.choice([4, 6, 8, 8, 8, 11])
    cells = particles / ppc
    a, b = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
    edge = cells ** (1 / 3)
    limit = 44 if material == "rubber" else 100
    nx, ny = (min(limit, max(4, round(edge * r))) for r in (a, b))
    nz = min(limit, max(4, int(cells / (nx * ny))))
    steps = max(1, min(20, int(work / (nx * ny * nz * ppc))))
    return {"path": path, "material": material, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "ppc": ppc,
            "steps": rng.randint(max(1, steps // 3), steps), "mls": path == "explicit" and rng.random() < 0.3}


# ------------------------------------------------------------------- inputs --
def _dt(case):
    return DT_EXPLICIT if case["path"] == "explicit" else SCENES[case["material"]][2]


def _inputs(case, seed):
    """Particles in motion: stratified positions, a smooth and a random part of the velocity with its gradient
    as C, and a smooth deformation of about two percent."""
    dx, log2, _, _, E, _ = SCENES[case["material"]]
    rng = np.random.default_rng([seed, 17])
    n = (case["nx"], case["ny"], case["nz"])
    size = np.array(n) * dx
    grid = np.stack(np.meshgrid(*[np.arange(c) for c in n], indexing="ij"), -1).reshape(-1, 3)
    x = np.repeat(grid, case["ppc"], 0) + rng.random((grid.shape[0] * case["ppc"], 3))
    if case["material"] in ("brittle", "cracking"):
        lo = 16 * dx + rng.random(3) * dx
    elif case["material"] == "foam":
        lo = np.array([0.5, 0.5, 0.5]) + np.array([-size[0] / 2, 2 * dx, -size[2] / 2]) + rng.random(3) * dx * [1, 0, 1]
    else:
        lo = np.array([5.0, 4.2, 5.0]) * dx + rng.random(3) * dx
    x = x * dx + lo
    P = x.shape[0]
    k = 2 * np.pi * rng.integers(1, 3, size=(3, 3)) / size * rng.choice([-1, 1], size=(3, 3))
    phase = rng.random((2, 3)) * 2 * np.pi
    arg = (x - lo) @ k.T
    wave = np.cos(arg + phase[0])
    amp = 0.3 * rng.uniform(0.5, 1.0, 3)
    v = amp * np.sin(arg + phase[0]) + rng.uniform(-0.2, 0.2, size=(P, 3))
    C = (amp * wave)[:, :, None] * k[None]
    # u_r = b_r sin(k_r . x): |grad u| of about 0.02
    b = 0.02 * rng.uniform(0.5, 1.0, 3) / np.linalg.norm(k, axis=1)
    F = np.eye(3) + (b * np.cos(arg + phase[1]))[:, :, None] * k[None]
    if case["material"] in ("brittle", "cracking"):
        v[:, 0] += 0.5 * (2 * (x[:, 0] - lo[0]) / size[0] - 1)
    if case["material"] == "foam":
        v[:, 1] -= math.sqrt(2 * 9.8 * 0.3)
    V0 = dx ** 3 / case["ppc"]
    out = {"x": x, "v": v, "C": C, "F": F, "lo": lo, "size": size, "V0": V0}
    if case["path"] == "reverse":
        out["E"] = np.exp(math.log(E) - REVERSE_SPREAD ** 2 / 2 + REVERSE_SPREAD * rng.standard_normal(P))
        out["gX"] = rng.standard_normal((P, 3)) / P
    return out


def _colliders(case, inp):
    """(kind, a, b, velocity): half spaces (origin, outward normal), boxes (corners), spheres (centre, radius)."""
    dx, log2, _, _, _, _ = SCENES[case["material"]]
    lo, size = inp["lo"], inp["size"]
    if case["material"] in ("brittle", "cracking"):
        hi, grip = lo + size, 3 * dx
        left = ("box", lo - 4 * dx, np.array([lo[0] + grip, hi[1] + 4 * dx, hi[2] + 4 * dx]), (-0.5, 0.0, 0.0))
        right = ("box", np.array([hi[0] - grip, lo[1] - 4 * dx, lo[2] - 4 * dx]), hi + 4 * dx, (0.5, 0.0, 0.0))
        return [left, right]
    if case["material"] == "foam":
        return [("sphere", np.array([0.5, 0.3, 0.5]), 0.2, (0.0, 0.0, 0.0)),
                ("half", np.array([0.0, 3 * dx, 0.0]), np.array([0.0, 1.0, 0.0]), (0.0, 0.0, 0.0))]
    if case["material"] == "rubber":
        return [("half", np.array([0.0, 3 * dx, 0.0]), np.array([0.0, 1.0, 0.0]), (0.0, 0.0, 0.0))]
    top = (1 << log2) * dx / 2
    walls = []
    for d in range(3):
        for s in (1.0, -1.0):
            o, nrm = np.zeros(3), np.zeros(3)
            o[d], nrm[d] = (3 * dx if s > 0 else top - 3 * dx), s
            walls.append(("half", o, nrm, (0.0, 0.0, 0.0)))
    return walls


def prepare(case, seed):
    dx, log2, dt, g, E, nu = SCENES[case["material"]]
    inp = _inputs(case, seed)
    sim = mpm.MpmSimulation(dx, gravity=(0.0, g, 0.0), precision=case["precision"], grid_log2=log2)
    h = sim.addParticles(inp["x"], inp["v"], RHO * inp["V0"], inp["V0"])
    m = case["material"]
    if m == "rubber":
        h.addFBasedMpmForce(mpm.FixedCorotated(E, nu))
        sim.switchLinearSolver(abi.CG)
        sim.newton_tolerance, sim.newton_max_iterations, sim.krylov_max_iterations = 1e-7, 10, 100
    elif m in ("brittle", "cracking"):
        h.addFBasedMpmForce(mpm.NeoHookeanBorden(E, nu))
        if m == "brittle":
            h.addRankineDamage(SIGMA_F, residual_phase=RESIDUAL)
        else:
            h.addFBasedMpmForceWithPhaseField(0.01, 0.5 * dx)
            sim.setPhaseFieldSolver(parabolic_M=1.0, lumping=True)
    else:
        model = mpm.StvkWithHenckyIsotropic(E, nu)
        h.addFBasedMpmForce(model)
        if m == "metal":
            h.addPlasticity(model, mpm.VonMisesStvkHencky(YIELD, 1e30, 0.0))
        elif m == "sand":
            h.addPlasticity(model, mpm.DruckerPragerStvkHencky(FRICTION, 1.0, 0.0, True))
        elif m == "foam":
            visc = 2 * E / (2 * (1 + nu)) * 0.05
            h.addFElasticNonequilibratedBasedMpmForce(mpm.StvkWithHencky(E, nu), visc, visc)
            sim.useAdmm(admm_max_iterations=20, rho_scale=0.8, global_tolerance=1e-8, local_tolerance=1e-8)
    for kind, a, b, vel in _colliders(case, inp):
        shape = {"half": lambda: mpm.HalfSpace(a, b), "box": lambda: mpm.AxisAlignedAnalyticBox(a, b),
                 "sphere": lambda: mpm.Sphere(a, b)}[kind]()
        obj = mpm.AnalyticCollisionObject(shape, abi.STICKY)
        obj.setTranslation((0.0, 0.0, 0.0), vel)
        sim.addCollisionObject(obj)
    if case["path"] == "explicit":
        sim.useExplicit(mls_mpm=case["mls"])
    state = {"sim": sim, "dt": _dt(case), "steps": case["steps"], "path": case["path"], "material": m}
    if case["path"] == "reverse":
        sim.newton_tolerance, sim.newton_max_iterations = 1e-12, 30
        sim.krylov_max_iterations, sim.krylov_tolerance = 500, 1e-30
        state.update(rollout=rollout.Rollout(sim, nu, dt, case["steps"], checkpoint_every=2, tolerance=1e-10), E=inp["E"], v0=inp["v"],
                     gX=inp["gX"])
    else:
        sim.setParticles(C=inp["C"], F=inp["F"])
        sim.checkpointSave(0)
    return state


def run(state):
    sim = state["sim"]
    if state["path"] == "reverse":
        X = state["rollout"].run(state["E"], state["v0"])
        gE, gv = state["rollout"].backward(state["gX"])
        return {"X": X, "gE": gE, "gv": gv}
    sim.checkpointLoad(0)
    for _ in range(state["steps"]):
        rc = sim.advanceOneTimeStep(state["dt"])
        if rc not in (abi.OK, abi.CFL_VIOLATION):
            raise RuntimeError(f"substep status {rc}")
    out = sim.getParticles()
    if state["material"] == "brittle":
        out["c"] = sim.getDamage()
    elif state["material"] == "cracking":
        out["c"] = sim.getPhaseField()["c"]
    return out


def work(case):
    """Per substep the particle state (x, v, C, F) in and out with its constants, per product of the linear
    solves (a usual count of them for the path) x, Fn, F, V0 of every particle and 27 values of every node."""
    P = case["nx"] * case["ny"] * case["nz"] * case["ppc"]
    nodes = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
    w = 4 if case["precision"] == "mixed" else 8
    newton, products = {"newton": (3, 12), "explicit": (1, 0), "admm": (20, 600), "reverse": (4 * 3, 100 * 3)}[case["path"]]
    if case["material"] == "rubber" and case["path"] == "newton":
        newton, products = 3, 30
    reads = P * 24 * 8 + (P * 8 if case["material"] in ("brittle", "cracking") else 0)
    per_step = P * (48 + 8) * 8 + products * ((7 if case["path"] == "admm" else 22) * w * P + 27 * 8 * nodes)
    flops = P * (3000 + newton * 3000 + products * (700 if case["path"] == "admm" else 1600))
    return {"bytes": float(case["steps"] * per_step + reads), "flops": float(case["steps"] * flops)}


def tolerance(case):
    """About four times what was measured.  Mixed Hencky materials keep FP32 noise of the strains (yielding particles
    sit on the surface): 2e-4 off `exact` in C after 20 substeps, 6e-5 between repeats (worst value 7e-4); the other
    mixed paths 3e-6 and 3e-6 (7e-5); fp64 7e-13 and 7e-14 (4e-12), where a converged solve amplifies it most."""
    if case["path"] == "reverse":
        return {"rel": 1e-5, "max": 1e-3} if case["precision"] == "mixed" else {"rel": 1e-8, "max": 1e-6}
    if case["precision"] == "fp64":
        return {"rel": 1e-11, "max": 1e-9}
    return {"rel": 1e-3, "max": 1e-2} if case["material"] in ("elastic", "metal", "sand") else {"rel": 2e-5, "max": 5e-4}


# -------------------------------------------------------------------- exact --
def exact(case, seed):
    """The substeps in 64 bits on plain torch tensors, for the Newton and explicit paths.  The ADMM local solves,
    the phase-field equation and the reverse sweep have no short restatement."""
    if case["path"] not in ("newton", "explicit") or case["material"] == "cracking":
        return None
    s = _Exact(case, _inputs(case, seed))
    for n in range(case["steps"]):
        s.substep(n * s.dt)
    out = {k: getattr(s, k).cpu().numpy() for k in ("X", "V", "C", "F")}
    if case["material"] == "brittle":
        out["c"] = s.c.cpu().numpy()
    return out


def _det(A):
    return (A[:, 0] * torch.linalg.cross(A[:, 1], A[:, 2])).sum(1)


def _cofactor(A):
    r = [A[:, 0], A[:, 1], A[:, 2]]
    return torch.stack([torch.linalg.cross(r[1], r[2]), torch.linalg.cross(r[2], r[0]), torch.linalg.cross(r[0], r[1])], 1)


def _svd(F):
    """F = U diag(s) V^T of 3x3 matrices with det > 0, by one-sided Jacobi rotations of the columns; s descends."""
    A, V = F.clone(), torch.eye(3, dtype=F.dtype, device=F.device).expand_as(F).clone()
    for _ in range(8):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            a, b = A[:, :, p], A[:, :, q]
            aa, bb, ab = (a * a).sum(1), (b * b).sum(1), (a * b).sum(1)
            z = (bb - aa) / torch.where(ab == 0, torch.ones_like(ab), 2 * ab)
            t = torch.where(z < 0, -1.0, 1.0) / (z.abs() + torch.sqrt(1 + z * z))
            t = torch.where(ab == 0, torch.zeros_like(t), t)
            c = 1 / torch.sqrt(1 + t * t)
            c, sn = c[:, None], (c * t)[:, None]
            for M in (A, V):
                mp, mq = M[:, :, p].clone(), M[:, :, q].clone()
                M[:, :, p], M[:, :, q] = c * mp - sn * mq, sn * mp + c * mq
    s, order = A.norm(dim=1).sort(1, descending=True)
    take = order[:, None, :].expand(-1, 3, -1)
    return torch.gather(A, 2, take) / s[:, None, :], s, torch.gather(V, 2, take)


class _Exact:
    def __init__(self, case, inp):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        self.case, self.inp, self.dev = case, inp, dev
        self.dx, _, _, gy, E, nu = SCENES[case["material"]]
        self.dt = _dt(case)
        self.g = t([0.0, gy, 0.0])
        self.mu, self.lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        self.kappa = 0.666666 * self.mu + self.lam
        self.V0, self.mass = inp["V0"], RHO * inp["V0"]
        self.X, self.V, self.C, self.F = (t(inp[k]) for k in ("x", "v", "C", "F"))
        P = self.X.shape[0]
        self.gd = torch.ones(P, dtype=torch.float64, device=dev)
        self.c = torch.ones_like(self.gd)
        self.logJp = torch.zeros_like(self.gd)
        self.t = t

    # transfers
    def bin(self):
        base = torch.floor(self.X / self.dx - 0.5)
        d = self.X / self.dx - base
        w = torch.stack([0.5 * (1.5 - d) ** 2, 0.75 - (d - 1) ** 2, 0.5 * (d - 0.5) ** 2], 2)
        dw = torch.stack([d - 1.5, -2 * (d - 1), d - 0.5], 2) / self.dx
        wx, wy, wz = w[:, 0], w[:, 1], w[:, 2]
        prod = lambda a, b, c: (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(-1, 27)  # noqa: E731
        self.w = prod(wx, wy, wz)
        self.dw = torch.stack([prod(dw[:, 0], wy, wz), prod(wx, dw[:, 1], wz), prod(wx, wy, dw[:, 2])], 2)
        o = torch.arange(3, device=self.dev)
        off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(27, 3)
        node = base.long()[:, None, :] + off[None]
        key = (node[..., 0] * 4096 + node[..., 1]) * 4096 + node[..., 2]
        ids, self.idx = torch.unique(key, return_inverse=True)
        self.xn = torch.stack([ids // (4096 * 4096), ids // 4096 % 4096, ids % 4096], 1).double() * self.dx
        self.rel = node.double() * self.dx - self.X[:, None, :]
        self.nn = ids.numel()

    def scatter(self, val):
        out = torch.zeros((self.nn,) + val.shape[2:], dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.idx.reshape(-1), val.reshape((-1,) + val.shape[2:]))

    def grad(self, x):  # sum_i x_i grad w_i^T
        return torch.einsum("pnr,pnc->prc", x[self.idx], self.dw)

    def force(self, S):  # -sum_p S grad w
        return -self.scatter(torch.einsum("prc,pnc->pnr", S, self.dw))

    # constitutive models
    def stress(self, F):
        """P(F), and what dP needs."""
        mu, lam = self.mu, self.lam
        if self.case["material"] in ("brittle", "cracking"):
            J = _det(F)
            FinvT = _cofactor(F) / J[:, None, None]
            B = F @ F.transpose(1, 2)
            tr = B.diagonal(dim1=1, dim2=2).sum(1)
            eye = torch.eye(3, dtype=F.dtype, device=F.device)
            td = (mu * J ** (-2.0 / 3.0))[:, None, None] * (B - tr[:, None, None] / 3 * eye)
            tv = (J * self.kappa / 2 * (J - 1 / J))[:, None, None] * eye
            gd = self.gd[:, None, None]
            tau = torch.where((J >= 1)[:, None, None], gd * (td + tv), gd * td + tv)
            return tau @ FinvT, (F, FinvT, J)
        U, s, V = _svd(F)
        if self.case["material"] == "rubber":
            J = s.prod(1, keepdim=True)
            psi = 2 * mu * (s - 1) + lam * (J - 1) * J / s
        else:
            L = s.log()
            psi = (2 * mu * L + lam * L.sum(1, keepdim=True)) / s
        return (U * psi[:, None, :]) @ V.transpose(1, 2), (U, s, V, psi)

    def dstress(self, aux, dF):
        mu, lam = self.mu, self.lam
        if self.case["material"] in ("brittle", "cracking"):
            F, FinvT, J = aux
            J = J[:, None, None]
            m = mu * J ** (-2.0 / 3.0)
            FF = (F * F).sum((1, 2), keepdim=True)
            a = (FinvT * dF).sum((1, 2), keepdim=True)
            b = (F * dF).sum((1, 2), keepdim=True)
            dFinvT = -FinvT @ dF.transpose(1, 2) @ FinvT
            # P_dev = m (F - |F|^2/3 F^-T), P_vol = kappa/2 (J^2 - 1) F^-T
            dev = -2.0 / 3.0 * m * a * (F - FF / 3 * FinvT) + m * (dF - 2.0 / 3.0 * b * FinvT - FF / 3 * dFinvT)
            vol = self.kappa * J * J * a * FinvT + self.kappa / 2 * (J * J - 1) * dFinvT
            gd = self.gd[:, None, None]
            return torch.where(J >= 1, gd * (dev + vol), gd * dev + vol)
        U, s, V, psi = aux
        D = U.transpose(1, 2) @ dF @ V
        K = torch.empty_like(D)
        d = D.diagonal(dim1=1, dim2=2)
        rubber = self.case["material"] == "rubber"
        if rubber:
            J = s.prod(1)
            co = J[:, None] / s
        else:
            L = s.log()
            S = L.sum(1)
        for i in range(3):
            acc = 0
            for j in range(3):
                if rubber:
                    h = 2 * mu + lam * co[:, i] ** 2 if i == j else lam * s[:, 3 - i - j] * (2 * J - 1)
                else:
                    h = ((2 * mu + lam) * (1 - L[:, i]) - lam * (S - L[:, i])) / s[:, i] ** 2 if i == j else lam / (s[:, i] * s[:, j])
                acc = acc + h * d[:, j]
            K[:, i, i] = acc
        for i, j in ((0, 1), (0, 2), (1, 2)):
            if rubber:
                m = 2 * mu - lam * (J - 1) * s[:, 3 - i - j]
            else:
                r = s[:, i] / s[:, j] - 1
                l1p = torch.where(r.abs() < 1e-6, torch.ones_like(r), torch.log1p(r) / torch.where(r == 0, torch.ones_like(r), r))
                m = -(lam * S + 2 * mu * (L[:, j] - l1p)) / (s[:, i] * s[:, j])
            p = (psi[:, i] + psi[:, j]) / (s[:, i] + s[:, j])
            K[:, i, j] = ((m + p) * D[:, i, j] + (m - p) * D[:, j, i]) / 2
            K[:, j, i] = ((m - p) * D[:, i, j] + (m + p) * D[:, j, i]) / 2
        return U @ K @ V.transpose(1, 2)

    def damage(self):
        F = self.F
        J = _det(F)
        B = F @ F.transpose(1, 2)
        tr = B.diagonal(dim1=1, dim2=2).sum(1)
        eye = torch.eye(3, dtype=F.dtype, device=F.device)
        cauchy = ((self.mu * J ** (-2.0 / 3.0))[:, None, None] * (B - tr[:, None, None] / 3 * eye)
                  + (J * self.kappa / 2 * (J - 1 / J))[:, None, None] * eye) / J[:, None, None]
        q = cauchy.diagonal(dim1=1, dim2=2).sum(1) / 3
        D = cauchy - q[:, None, None] * eye
        p = torch.sqrt((D * D).sum((1, 2)) / 6)
        r = (_det(D / p[:, None, None]) / 2).clamp(-1, 1)
        smax = q + 2 * p * torch.cos(torch.acos(r) / 3)
        self.c = torch.where(smax > SIGMA_F, torch.minimum(self.c, SIGMA_F / smax), self.c)
        self.gd = self.c ** 2 * (1 - RESIDUAL) + RESIDUAL

    def plasticity(self):
        m = self.case["material"]
        if m not in ("metal", "sand"):
            return
        U, s, V = _svd(self.F)
        mu, lam = self.mu, self.lam
        e = s.clamp(min=1e-4).log()
        if m == "metal":
            h = e - e.sum(1, keepdim=True) / 3
            hn = h.norm(dim=1, keepdim=True)
            dg = hn - YIELD / (2 * mu)
            out = torch.exp(e - dg / hn * h)
            new = (U * out[:, None, :]) @ V.transpose(1, 2)
            self.F = torch.where((dg > 0)[:, :, None], new, self.F)
            return
        sin = math.sin(FRICTION / 180.0 * 3.141592653)
        alpha = math.sqrt(2.0 / 3.0) * 2 * sin / (3 - sin)
        es = e.sum(1, keepdim=True)
        tr = es + self.logJp[:, None]
        h = e - tr / 3
        hn = h.norm(dim=1, keepdim=True)
        dg = hn + (3 * lam + 2 * mu) / (2 * mu) * tr * alpha
        out = torch.exp(torch.where(dg <= 0, e, e - dg / hn * h))
        out = torch.where(tr >= 0, torch.ones_like(out), out)
        self.logJp = torch.where(tr[:, 0] >= 0, es[:, 0] + self.logJp, torch.zeros_like(self.logJp))
        self.F = (U * out[:, None, :]) @ V.transpose(1, 2)

    # colliders (sticky)
    def inside(self, x, time, only=None):
        hit = torch.zeros(x.shape[0], dtype=torch.bool, device=self.dev)
        vel = torch.zeros_like(x)
        for kind, a, b, v in _colliders(self.case, self.inp):
            y = x - self.t(v) * time
            if kind == "half":
                n = ((y - self.t(a)) @ self.t(b)) <= 0
            else:
                n = (((y - self.t((a + b) / 2)).abs() - self.t((b - a) / 2)) <= 0).all(1)
            vel = torch.where((n & ~hit)[:, None], self.t(v).expand_as(x), vel)
            hit |= n
        return hit, vel

    def substep(self, time):
        dt = self.dt
        self.bin()
        self.m = self.scatter(self.w * self.mass)
        aff = self.V[:, None, :] + torch.einsum("prc,pnc->pnr", self.C, self.rel)
        vn = self.scatter((self.w * self.mass)[..., None] * aff) / self.m[:, None]
        if self.case["path"] == "explicit":
            P, _ = self.stress(self.F)
            tau = self.V0 * P @ self.F.transpose(1, 2)
            if self.case["mls"]:
                f = -self.scatter(torch.einsum("prc,pnc->pnr", tau, self.rel) * (self.w * 4 / self.dx ** 2)[..., None])
            else:
                f = self.force(tau)
            vs = vn + self.g * dt + f * dt / self.m[:, None]
            hit, vel = self.inside(self.xn, time)
            vs = torch.where(hit[:, None], vel, vs)
            for _, a, b, _ in _colliders(self.case, self.inp):  # trial collision with the half spaces
                phi = (self.xn + dt * vs - self.t(a)) @ self.t(b)
                vs = torch.where(((phi <= 0) & ~hit)[:, None], vs - (phi / dt)[:, None] * self.t(b), vs)
        else:
            if self.case["material"] == "brittle":
                self.damage()
            vs = self.newton(vn, time)
        wv = self.w[..., None] * vs[self.idx]
        self.V = wv.sum(1)
        B = torch.einsum("pnr,pnc->prc", wv, self.rel)
        C = B * (4 / self.dx ** 2)
        gv = C if self.case["mls"] else self.grad(vs)
        self.C = C
        self.X = self.X + dt * self.V
        self.F = self.F + dt * gv @ self.F
        self.plasticity()

    def newton(self, vn, time):
        dt, m = self.dt, self.m[:, None]
        rubber = self.case["material"] == "rubber"
        tol, nmax, kmax = (1e-7, 10, 100) if rubber else (1e-5, 3, 20)
        eps = np.finfo(np.float64 if self.case["precision"] == "fp64" else np.float32).eps
        abs_tol = 16 * float(eps) if rubber else 1.0
        hit, vel = self.inside(self.xn, time)
        free = (~hit)[:, None].double()
        dv = torch.where(hit[:, None], vel - vn, (self.g * dt).expand_as(vn))
        Fn = self.F
        for _ in range(nmax):
            P, aux = self.stress(Fn + dt * self.grad(vn + dv) @ Fn)
            r = free * (dt * self.g * m + dt * self.force(self.V0 * P @ Fn.transpose(1, 2)) - m * dv)
            norm = math.sqrt(float((r * r / m).sum()))
            if norm < tol:
                break
            lt = min(min(0.5, math.sqrt(max(norm, tol))) * norm, abs_tol)
            if norm < lt:
                continue

            def A(z):
                dP = self.dstress(aux, self.grad(z) @ Fn)
                return free * (m * z - dt * dt * self.force(self.V0 * dP @ Fn.transpose(1, 2)))
            dv = dv + (self.cg if rubber else self.minres)(A, r, norm, lt, kmax)
        return vn + dv

    def cg(self, A, r, norm, lt, kmax):
        m = self.m[:, None]
        x = torch.zeros_like(r)
        q = r / m
        p, zr = q, norm * norm
        for _ in range(kmax):
            t = A(p)
            alpha = zr / float((p * t).sum())
            x = x + alpha * p
            r = r - alpha * t
            q = r / m
            z1 = float((q * r).sum())
            p = q + z1 / zr * p
            zr = z1
            if math.sqrt(zr) < lt:
                break
        return x

    def minres(self, A, r, norm, lt, kmax):
        m = self.m[:, None]
        x, q0, m1, m2 = (torch.zeros_like(r) for _ in range(4))
        beta, q, z = norm, r / norm, r / m / norm
        c1, s1, c2, s2, rhs = 1.0, 0.0, 1.0, 0.0, norm
        for _ in range(kmax):
            w = A(z)
            alpha = float((w * z).sum())
            qn = w - alpha * q - beta * q0
            zn = qn / m
            bn = math.sqrt(max(float((zn * qn).sum()), 0.0))
            e, d = -s2 * beta, c2 * beta
            delta, t0 = c1 * d - s1 * alpha, s1 * d + c1 * alpha
            sd = math.hypot(t0, bn)
            c, sn = (t0 / sd, -bn / sd) if sd else (1.0, 0.0)
            gamma = c * t0 - sn * bn
            mk = (z - delta * m1 - e * m2) / gamma
            x = x + c * rhs * mk
            rhs = sn * rhs
            if abs(rhs) < lt or bn == 0:
                break
            c2, s2, c1, s1 = c1, s1, c, sn
            m2, m1 = m1, mk
            q0, q, z, beta = q, qn / bn, zn / bn, bn
        return x
