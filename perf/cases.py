"""The workloads this library is timed on: what a user's program does with it, through its public entry points.

Simulations. One pass is one output interval of a program: the initial conditions go in from pinned host
memory, the solver takes a few steps (one captured graph per step), the energies are printed where a run
monitors them, and the state comes back to the host. The context (device buffers, launch shapes) is made
once in prepare(), as a program keeps it.

Network. One pass is one forward over a particle set, or one minibatch gradient of the training loop.

exact() restates each path in 64-bit torch (all pairs, no neighbour structures), from the same inputs.
"""

import math
import os

import numpy as np
import torch

import grasph2_b200
from grasph2_b200 import ics
from grasph2_b200.mlp import MLP, SHAPES, init_params
from grasph2_b200.params import config0_params, config2_params, impact_params, make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer, Ensemble

SURROGATE_FILE = os.path.join(os.path.dirname(os.path.abspath(grasph2_b200.__file__)), "data", "surrogate_impact_n262144")
FLAG_DEAL_WITH_NO_PARTNERS = 1 << 3
ENERGIES = ("e_kin", "e_grav", "e_int", "e_shear", "mass")  # momenta vanish in these centre-of-mass frames
ENSEMBLE_SIZES = (1024, 32768)


# ---- the cases ----------------------------------------------------------------------------------------
def _sim(name, path, n, steps, accum="plain", precision="single", masses="equal", energies=False):
    c = {"path": path, "n": n, "steps": steps, "accum": accum, "precision": precision, "masses": masses,
         "energies": energies}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small star cluster between two outputs: twenty short launches in a row, latency counts
        _sim("nbody-4096", "nbody", 4096, 20),
        # a cluster with a stellar mass function, an odd particle number, compensated sums
        _sim("nbody-100003-comp", "nbody", 100003, 2, accum="compensated", masses="spread"),
        # the Plummer sphere at the largest single-GPU size: one step is already a third of a second
        _sim("nbody-1048576", "nbody", 1048576, 1),
        # the small fluid sphere (liquid EOS, summed density): the smallest SPH run, launches count
        _sim("fluid-4096", "fluid", 4096, 20, energies=True),
        # the elastic-plastic impact of two spheres, the library's ordinary SPH + gravity run
        _sim("impact-65536", "impact", 65536, 10, energies=True),
        # the reference's shipped settings: a rotating rubble body, Mohr-Coulomb, Balsara switch,
        # integrated density, variable time step
        _sim("rubble-16384", "rubble", 16384, 10, energies=True),
        # the double-precision switch: a small fluid sphere, and an impact of odd size
        _sim("double-fluid-4096", "fluid", 4096, 5, precision="double", energies=True),
        _sim("double-impact-30011", "impact", 30011, 2, precision="double", energies=True),
        # a parameter study: 512 spheres of 1,024 to 32,768 particles advanced together
        {"name": "ensemble-512", "path": "ensemble", "n": 512, "steps": 2, "accum": "plain"},
        # the learned surrogate: two proposals of eight substeps each on the large impact
        {"name": "surrogate-262144", "path": "surrogate", "n": 262144, "steps": 2},
        # the surrogate's network over every particle of that impact
        {"name": "mlp-forward-262144", "path": "mlp_forward", "n": 262144},
        # the gradient of one training minibatch (the training script's batch), read back by the program
        {"name": "mlp-gradient-65536", "path": "mlp_gradient", "n": 65536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["nbody", "nbody", "fluid", "impact", "impact", "rubble", "double", "double", "ensemble",
                       "surrogate", "mlp_forward", "mlp_gradient"])
    accum = rng.choice(["plain", "plain", "compensated"])
    if path == "nbody":
        n = _log_int(rng, 1000, 600000)
        return _sim(None, path, n, rng.randint(1, 1 + min(19, 200000 // n)), accum=accum,
                    masses=rng.choice(["equal", "spread"]))
    if path == "fluid":
        n = _log_int(rng, 1000, 60000)
        return _sim(None, path, n, rng.randint(1, 20), accum=accum, energies=rng.random() < 0.5)
    if path == "impact":
        n = _log_int(rng, 4000, 250000)
        return _sim(None, path, n, rng.randint(1, 2 + min(18, 600000 // n)), accum=accum, energies=rng.random() < 0.5)
    if path == "rubble":
        return _sim(None, path, _log_int(rng, 2000, 65536), rng.randint(1, 20), accum=accum, energies=rng.random() < 0.5)
    if path == "double":
        kind = rng.choice(["nbody", "fluid", "impact", "rubble"])
        n = _log_int(rng, 1000, 40000)
        return _sim(None, kind, n, rng.randint(1, 3), precision="double",
                    masses=rng.choice(["equal", "spread"]) if kind == "nbody" else "equal",
                    energies=rng.random() < 0.5)
    if path == "ensemble":
        return {"path": path, "n": _log_int(rng, 8, 400), "steps": rng.randint(1, 2), "accum": accum}
    if path == "surrogate":
        return {"path": path, "n": _log_int(rng, 30000, 262144), "steps": rng.randint(1, 2)}
    if path == "mlp_forward":
        return {"path": path, "n": _log_int(rng, 1000, 1000000)}
    return {"path": path, "n": _log_int(rng, 1000, 262144)}


# ---- inputs -------------------------------------------------------------------------------------------
def _split(n):
    big = round(n * 8 / 9)  # radii 1 and 0.5 at equal number density
    return big, n - big


def _params(case):
    path, n = case["path"], case["n"]
    if path == "nbody":
        return config2_params()
    if path == "fluid":
        return config0_params()
    if path in ("impact", "surrogate"):
        return impact_params(*_split(n))
    if path == "ensemble":
        p = config0_params()
        p.flags |= FLAG_DEAL_WITH_NO_PARTNERS  # h is fixed, so the smallest spheres are sparsely sampled
        return p
    h = 0.25 * n ** (-1.0 / 3.0)  # the shipped settings at another particle count (radius 0.1, mass 1)
    return make_params(H=h)


def _unit_sphere(rng, n):
    """A settled sphere: the n points of a jittered cubic lattice that are nearest to the origin."""
    d = (4.0 / 3.0 * math.pi / n) ** (1.0 / 3.0)
    k = np.arange(-int(1.1 / d) - 2, int(1.1 / d) + 3)
    x = np.stack(np.meshgrid(k, k, k, indexing="ij"), axis=-1).reshape(-1, 3)
    x = (x + rng.uniform(0.0, 1.0, 3)) * d
    r2 = (x * x).sum(1)
    x = x[np.argpartition(r2, n)[:n]] + rng.uniform(-0.2 * d, 0.2 * d, (n, 3))
    return rng.permutation(x - x.mean(0))


def _state(case, seed):
    """The initial conditions (float64 arrays by attribute) and, for the ensemble, the sizes."""
    path, n = case["path"], case["n"]
    rng = np.random.default_rng(1000003 + 7919 * seed)
    if path == "nbody":
        st = ics.plummer_sphere(n, seed=seed)
        out = {k: st[k] for k in ("pos", "mass", "vel")}
        if case["masses"] == "spread":  # power law of index -2.35 between 0.1 and 20, total mass 1
            u = rng.uniform(0.0, 1.0, n)
            m = (0.1 ** -1.35 + u * (20.0 ** -1.35 - 0.1 ** -1.35)) ** (-1.0 / 1.35)
            out["mass"] = m / m.sum()
        return out, None
    if path in ("impact", "surrogate"):
        st = ics.two_sphere_impact(*_split(n), v_rel=0.5, y_offset=0.3, seed=seed)
    elif path == "rubble":
        st = ics.uniform_sphere(n, radius=0.1, rho0=1.0 / (4.0 / 3.0 * math.pi * 0.1 ** 3), omega=(0.0, 0.0, 10.0),
                                seed=seed)
    else:  # fluid spheres with a rigid rotation: one, or an ensemble whose sizes go with their number
        lo, hi = ENSEMBLE_SIZES
        sizes = np.array([n])
        if path == "ensemble":
            u = np.random.default_rng(n).uniform(math.log(lo), math.log(hi + 1), n)
            sizes = np.floor(np.exp(u)).astype(np.int64).clip(lo, hi)
        x = np.concatenate([_unit_sphere(rng, int(k)) for k in sizes])
        om = np.repeat(rng.uniform(0.0, 0.5, len(sizes)), sizes)
        v = np.stack([-om * x[:, 1], om * x[:, 0], np.zeros_like(om)], axis=1)
        st = {"pos": x, "mass": np.repeat(1.0 / sizes, sizes), "vel": v, "density": np.full(len(x), 0.239)}
        return st, sizes if path == "ensemble" else None
    return {k: st[k] for k in ("pos", "mass", "vel", "density", "dstress")}, None


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=torch.cuda.is_available())
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t.numpy()


def _results(case):
    """The attributes a program reads back."""
    path = case["path"]
    if path == "nbody":
        return ["pos", "vel", "acc"]
    if path in ("fluid", "ensemble"):
        return ["pos", "vel", "acc", "density"]
    return ["pos", "vel", "acc", "density", "dstress"]


def _x(case, seed):
    g = torch.Generator(device="cuda").manual_seed(2 * seed + 1)
    return torch.randn(case["n"], 32, device="cuda", generator=g)


def _target(case, seed):
    g = torch.Generator(device="cuda").manual_seed(2 * seed + 2)
    return torch.randn(case["n"], 13, device="cuda", generator=g)


def prepare(case, seed):
    path, n = case["path"], case["n"]
    s = {"path": path, "case": case}
    if path == "mlp_forward":
        s.update(net=MLP(init_params(seed)), x=_x(case, seed), y=torch.empty(n, 13, device="cuda"))
        return s
    if path == "mlp_gradient":
        s.update(net=MLP(init_params(seed)), x=_x(case, seed), t=_target(case, seed), w=torch.ones(13, device="cuda"))
        return s
    st, sizes = _state(case, seed)
    double = case.get("precision") == "double"
    opt = make_options(accum=case.get("accum", "plain"), precision=case.get("precision", "single"))
    total = n if sizes is None else int(sizes.sum())
    s["attrs"] = _results(case)
    if double:  # the reference's DOUBLE_PRECISION host buffers
        s["state"] = {k: np.ascontiguousarray(v, dtype=np.float64) for k, v in st.items()}
    else:
        s["state"] = {k: _pinned(v) for k, v in st.items()}
        shape = {"density": (total,), "dstress": (total, 3, 3)}
        s["out"] = {k: _pinned(np.zeros(shape.get(k, (total, 3)), np.float32)) for k in s["attrs"]}
    s["pb"] = Ensemble(_params(case), sizes, opt) if path == "ensemble" else DeviceParticleBuffer(_params(case), n, opt)
    if path == "surrogate":
        from grasph2_b200.surrogate import Surrogate
        s["sur"] = Surrogate.load(SURROGATE_FILE + ".gsur")
    return s


# ---- one pass -----------------------------------------------------------------------------------------
def run(s):
    path, case = s["path"], s["case"]
    if path == "mlp_forward":
        s["net"].forward(s["x"], s["y"], case["n"])
        return s["y"]
    if path == "mlp_gradient":
        grad, loss = s["net"].gradient(s["x"], s["t"], s["w"], case["n"])
        return {"grad": grad, "loss": loss}
    pb = s["pb"]
    double = case.get("precision") == "double"
    (pb.upload_f64 if double else pb.upload)(s["state"])
    if path == "surrogate":
        for _ in range(case["steps"]):
            s["sur"].propose(pb)
    else:
        pb.step(case["steps"])
    out = {}
    if case.get("energies"):
        e = pb.diagnostics()
        out.update({k: e[k] for k in ENERGIES})
    if double:
        out.update(pb.download_f64(s["attrs"]))
    else:
        out.update(pb.download(s["attrs"], out=s["out"]))
    return out


# ---- what one pass cannot do without --------------------------------------------------------------------
# per unordered pair of the gravity sum: the separation 3, r^2 6, 1/r^3 3, both masses 2, both sums 12
PAIR = 26
# per particle and neighbour: the density sum 10 (+ 8 for the distance); the stress rate, acceleration and
# artificial viscosity of a solid 160, of a fluid 60
NEIGHBOUR = {"fluid": 78, "ensemble": 78, "impact": 178, "surrogate": 178, "rubble": 178}


def _neighbours(path, n):
    """Mean number of particles within h of one, for n particles spread evenly."""
    if path in ("impact", "surrogate"):
        return 4.0 / 3.0 * math.pi * 2.5 ** 3
    if path == "rubble":
        return 2.5 ** 3
    return n * 0.15 ** 3


def work(case):
    path, n = case["path"], case["n"]
    weights = sum(int(np.prod(s)) for s in SHAPES)
    mul = sum(int(np.prod(s)) for s in SHAPES if len(s) == 2)
    if path == "mlp_forward":
        return {"bytes": 4 * (n * (32 + 13) + weights), "flops": 2.0 * n * mul}
    if path == "mlp_gradient":  # forward, the weights' gradient, and the activations' (not the input's)
        return {"bytes": 4 * (n * (32 + 13) + 2 * weights), "flops": 2.0 * n * (3 * mul - 32 * 128)}
    if path == "ensemble":
        lo, hi = ENSEMBLE_SIZES
        ln = math.log(hi / lo)
        total, pairs = n * (hi - lo) / ln, n * (hi ** 2 - lo ** 2) / (2 * ln) / 2  # log-uniform sizes
        nb = pairs * 2 * 0.15 ** 3
    else:
        total, pairs = n, n * (n - 1) / 2.0
        nb = 0.0 if path == "nbody" else n * _neighbours(path, n)
    inputs = {"nbody": 7, "fluid": 8, "ensemble": 8}.get(path, 17)
    outputs = {"nbody": 9, "fluid": 10, "ensemble": 10}.get(path, 19)
    size = 8 if case.get("precision") == "double" else 4
    flops = case["steps"] * (PAIR * pairs + nb * NEIGHBOUR.get(path, 0))
    if path == "surrogate":
        flops += case["steps"] * n * 2.0 * mul
    if case.get("energies"):
        flops += 12 * pairs
    return {"bytes": total * size * (inputs + outputs), "flops": flops}


# ---- the same in 64 bits ----------------------------------------------------------------------------------
def exact(case, seed):
    path = case["path"]
    if path == "mlp_forward":
        return _net(init_params(seed), _x(case, seed).double())[0]
    if path == "mlp_gradient":
        x, t = _x(case, seed).double(), _target(case, seed).double()
        y, ws = _net(init_params(seed), x, grad=True)
        loss = ((y - t) ** 2).sum() / case["n"]
        g = torch.autograd.grad(loss, ws)
        return {"grad": torch.cat([v.reshape(-1) for v in g]).cpu().numpy(), "loss": float(loss)}
    st, sizes = _state(case, seed)
    if case.get("precision") != "double":
        st = {k: v.astype(np.float32) for k, v in st.items()}
    st = {k: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).cuda() for k, v in st.items()}
    if path == "ensemble":
        off = np.concatenate([[0], np.cumsum(sizes)])
        parts = [_simulate(case, {k: v[a:b] for k, v in st.items()})[0] for a, b in zip(off[:-1], off[1:])]
        return {k: torch.cat([q[k] for q in parts]).cpu().numpy() for k in _results(case)}
    out, sim = _simulate(case, st)
    got = sim.energies(out) if case.get("energies") else {}
    got.update({k: out[k].cpu().numpy() for k in _results(case)})
    if path == "surrogate":  # from a stress-free start the network's 16-bit correction is most of it
        got["dstress"] = None
    return got


def _net(flat, x, grad=False):
    ws, o = [], 0
    for shape in SHAPES:
        k = int(np.prod(shape))
        ws.append(torch.from_numpy(flat[o:o + k].astype(np.float64)).cuda().reshape(shape).requires_grad_(grad))
        o += k
    h = x
    for k in range(0, 8, 2):
        h = h @ ws[k].T + ws[k + 1]
        if k < 6:
            h = torch.nn.functional.silu(h)
    return h, ws


class _Physics:
    """computeDerivatives and the leapfrog over all pairs, 64-bit."""

    def __init__(self, p):
        self.p = p
        f = p.flags
        (self.grav, self.sph, self.int_rho, self.floor, self.solid, self.variable, self.acc_crit, self.vel_crit,
         self.mises, self.mc) = [bool(f >> b & 1) for b in range(10)]
        self.av, self.balsara = bool(f >> 13 & 1), bool(f >> 14 & 1)
        self.dt = 0.0

    def pairwise(self, x, fn):
        """fn(rows a, b; r^2 of rows a..b against every particle) for blocks of rows."""
        c = x - x.mean(0)
        sq = (c * c).sum(1)
        right = torch.cat([-2.0 * c, torch.ones_like(sq)[:, None], sq[:, None]], 1).T.contiguous()
        step = max(1, min(len(x), 2 ** 25 // len(x)))
        for a in range(0, len(x), step):
            b = min(len(x), a + step)
            fn(a, b, torch.cat([c[a:b], sq[a:b, None], torch.ones_like(sq[a:b])[:, None]], 1) @ right)

    def gravity(self, x, m):
        acc = torch.empty_like(x)
        src = torch.cat([m[:, None] * x, m[:, None]], 1)

        def block(a, b, r2):
            s = r2.add_(self.p.grav_eps ** 2).rsqrt_()
            s = s.mul_(s * s) @ src
            acc[a:b] = s[:, :3] - x[a:b] * s[:, 3:]
        self.pairwise(x, block)
        return self.p.grav_G * acc

    def neighbours(self, x):
        """Index pairs (i, j) with 0 < r <= H."""
        H2, got = self.p.H ** 2, []

        def block(a, b, r2):
            i, j = torch.nonzero(r2 <= H2 * (1.0 + 1e-6) + 1e-12, as_tuple=True)
            got.append(torch.stack([i + a, j]))
        self.pairwise(x, block)
        i, j = torch.cat(got, 1)
        r2 = ((x[i] - x[j]) ** 2).sum(1)
        keep = (r2 > 0) & (r2 <= H2)
        return i[keep], j[keep]

    def sum(self, i, v, n):
        return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add_(0, i, v)

    def w(self, q):
        return torch.where(q < 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q) ** 3) * (8.0 / (math.pi * self.p.H ** 3))

    def dw(self, q):
        return torch.where(q < 0.5, 3 * q ** 2 - 2 * q, -(1 - q) ** 2) * (48.0 / (math.pi * self.p.H ** 4))

    def pressure(self, rho):
        p = self.p
        if self.solid:
            return p.bulk / p.dbulk_dp * ((rho / p.rho0) ** p.dbulk_dp - 1.0)
        return p.soundspeed ** 2 * (rho - p.rho0)

    def derivatives(self, s):
        p, n, x, m, v = self.p, len(s["mass"]), s["pos"], s["mass"], s["vel"]
        acc = self.gravity(x, m) if self.grav else torch.zeros_like(x)
        if self.sph:
            i, j = self.neighbours(x)
            d = x[i] - x[j]
            r = d.norm(dim=1)
            q = r / p.H
            if not self.int_rho:
                s["density"] = self.sum(i, m[j] * self.w(q), n)
                if self.floor:
                    s["density"] = torch.where(s["density"] < 0.001, 0.01 * p.rho0, s["density"])
            rho = s["density"]
            eye = torch.eye(3, dtype=x.dtype, device=x.device)
            sig = -self.pressure(rho)[:, None, None] * eye
            if self.solid:
                sig = sig + s["dstress"]
            sig = sig / (rho * rho)[:, None, None]
            g = (self.dw(q) / r)[:, None] * d
            vij = v[i] - v[j]
            if self.solid or self.int_rho or self.balsara:
                mr = m[j] / rho[j]
                L = self.sum(i, -mr[:, None, None] * vij[:, :, None] * g[:, None, :], n)  # dv_a / dx_b
                E, W = 0.5 * (L + L.transpose(1, 2)), 0.5 * (L - L.transpose(1, 2))
                div = L.diagonal(dim1=1, dim2=2).sum(1)
                if self.solid:
                    S = s["dstress"]
                    s["S_dt"] = 2 * p.shear * (E - div[:, None, None] * eye / 3) + S @ W.transpose(1, 2) + W @ S
                s["rho_dt"] = -rho * div
                curl = 2.0 * torch.stack([W[:, 2, 1], W[:, 0, 2], W[:, 1, 0]], 1).norm(dim=1)
                bal = div.abs() / (div.abs() + curl + 1e-4 * p.soundspeed / p.H)
            a = m[j][:, None] * torch.einsum("nab,nb->na", sig[i] + sig[j], g)
            vmax = torch.zeros(n, dtype=x.dtype, device=x.device)
            if self.av:
                w = (d * vij).sum(1) / r
                vsig = 2 * p.soundspeed - p.av_beta * w
                b = bal[i] + bal[j] if self.balsara else 2.0
                visc = -0.25 * b * p.av_alpha * w * vsig / (0.5 * (rho[i] + rho[j]))
                a = a - torch.where(w < 0, m[j] * visc, 0.0)[:, None] * g
                if self.balsara:
                    vmax = vmax.index_reduce_(0, i, torch.where(w < 0, vsig, 0.0), "amax")
            acc = acc + self.sum(i, a, n)
            s["vmax"] = vmax
        s["acc"] = acc

    def kick_drift(self, s, kick, dt):
        p = self.p
        s["vel"] = s["vel"] + kick * s["acc"]
        s["pos"] = s["pos"] + dt * s["vel"]
        if self.sph and self.int_rho:
            s["density"] = (s["density"] + dt * s["rho_dt"]).clamp(min=0.0)
        if self.sph and self.solid:
            s["dstress"] = s["dstress"] + dt * s["S_dt"]
            Y = p.tanfr * self.pressure(s["density"]) + p.cohesion if self.mc else p.Y
            if self.mc or self.mises:
                f = Y * Y / (1.5 * (s["dstress"] ** 2).sum((1, 2)))
                s["dstress"] = s["dstress"] * torch.where(f < 1.0, f, 1.0)[:, None, None]

    def step(self, s):
        p = self.p
        self.derivatives(s)
        if not self.variable:
            return self.kick_drift(s, p.fixed_dt, p.fixed_dt)
        s["vel"] = s["vel"] + 0.5 * self.dt * s["acc"]
        dt = p.max_dt
        if self.acc_crit:
            dt = min(dt, float(torch.sqrt(p.accel_accuracy * p.H / s["acc"].norm(dim=1)).min()))
        if self.vel_crit:
            dt = min(dt, float((p.velocity_accuracy * p.H / s["vmax"]).min()))
        self.dt = max(dt, p.min_dt)
        self.kick_drift(s, 0.5 * self.dt, self.dt)

    def energies(self, s):
        p, m = self.p, s["mass"]
        out = {k: 0.0 for k in ENERGIES}
        out["e_kin"] = float((0.5 * m * (s["vel"] ** 2).sum(1)).sum())
        out["mass"] = float(m.sum())
        phi = torch.empty_like(m)

        def block(a, b, r2):
            phi[a:b] = r2.add_(p.grav_eps ** 2).rsqrt_() @ m - m[a:b] / p.grav_eps
        self.pairwise(s["pos"], block)
        out["e_grav"] = float(-0.5 * p.grav_G * (m * phi).sum())
        if self.sph:
            rho = s["density"]
            u = torch.log(rho / p.rho0) + p.rho0 / rho - 1.0
            if self.solid:
                k = p.dbulk_dp
                if abs(k - 1.0) < 1e-12:
                    u = p.bulk / p.rho0 * u
                else:
                    u = p.bulk / k * ((rho ** (k - 1) - p.rho0 ** (k - 1)) / ((k - 1) * p.rho0 ** k) + 1 / rho - 1 / p.rho0)
                out["e_shear"] = float((m * (s["dstress"] ** 2).sum((1, 2)) / (4 * p.shear * rho)).sum())
            else:
                u = p.soundspeed ** 2 * u
            out["e_int"] = float((m * u).sum())
        return out

    def features(self, s):
        p, n, x, v = self.p, len(s["mass"]), s["pos"], s["vel"]
        i, j = self.neighbours(x)
        d, u = (x[j] - x[i]) / p.H, v[j] - v[i]
        w = (s["mass"][j] * self.w(d.norm(dim=1)) / p.rho0)[:, None]
        six = [0, 4, 8, 1, 2, 5]
        cols = [v, (s["density"] / p.rho0 - 1.0)[:, None], s["dstress"].reshape(n, 9)[:, six], self.sum(i, w, n),
                self.sum(i, w * d, n), self.sum(i, w * u, n),
                self.sum(i, w * (d[:, :, None] * d[:, None, :]).reshape(-1, 9)[:, six], n),
                self.sum(i, w * (u[:, :, None] * d[:, None, :]).reshape(-1, 9), n)]
        return torch.cat(cols, 1)

    def propose(self, s, model):
        """One K-substep proposal: the leapfrog with constant derivatives plus the network's correction."""
        K, dt = int(model["K"]), self.p.fixed_dt
        self.derivatives(s)
        f = (self.features(s) - model["in_mu"]) / model["in_sig"]
        c = model["out_mu"] + model["out_sig"] * _net(model["params"], f)[0]
        T = K * dt
        s["pos"] = s["pos"] + T * s["vel"] + 0.5 * K * (K + 1) * dt * dt * s["acc"] + c[:, 0:3]
        s["vel"] = s["vel"] + T * s["acc"] + c[:, 3:6]
        s["density"] = (s["density"] + c[:, 6]).clamp(min=0.0)
        S = s["dstress"] + T * s["S_dt"] + c[:, [7, 10, 11, 10, 8, 12, 11, 12, 9]].reshape(-1, 3, 3)
        f = self.p.Y ** 2 / (1.5 * (S ** 2).sum((1, 2)))
        s["dstress"] = S * torch.where(f < 1.0, f, 1.0)[:, None, None]


def _simulate(case, st):
    p = _params(case)
    if case.get("precision") != "double":  # the constants as single precision holds them
        for name, _ in p._fields_:
            if isinstance(getattr(p, name), float):
                setattr(p, name, float(np.float32(getattr(p, name))))
    sim, s = _Physics(p), dict(st)
    if case["path"] == "surrogate":
        z = np.load(SURROGATE_FILE + ".npz")
        model = {k: torch.from_numpy(z[k].astype(np.float64)).cuda() for k in ("in_mu", "in_sig", "out_mu", "out_sig")}
        model.update(K=z["K"], params=z["params"])
        for _ in range(case["steps"]):
            sim.propose(s, model)
    else:
        for _ in range(case["steps"]):
            sim.step(s)
    return s, sim
