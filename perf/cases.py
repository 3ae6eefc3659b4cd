"""What this framework is used for, as cases that can be timed and compared.

Every case is a stretch of a run loop through the public Python API: the
solver a program keeps (its grid, physics and storage format), advanced by a
number of lattice steps, then its diagnostics and fields read back, as the
driver does between its progress events.  The state goes on from pass to pass,
as a run's does.  Five kinds:

uniform  one cavity (CavitySolver.step, diag, fields), fixed-Cs or with the
         dynamic mixed-scale subgrid model
batch    many cavities of uneven size and Rayleigh number in lockstep
         (CavityBatch.step, fields), after the library's own autotuning
adjoint  init_from_fields, then the gradient of the time-averaged hot-wall
         Nusselt number w.r.t. the wall profile and Cs (adjoint_nusselt)
octree   the block-refined cavity (OctreeSolver.step_cavity, diag, level),
         with or without the dynamic model on every level

exact() restates the reference's time step in FP64 torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

PR, PR_T, UTARGET, T_COLD = 0.71, 0.9, 0.02, -0.5
BATCH_GRIDS = ((64, 256), (96, 384), (128, 512))
# bytes of one stored population and of the Guo force per node
STORE = {"f64": (8, 8), "f32": (4, 4), "f16": (2, 4), "bf16": (2, 4), "f16g": (2, 4), "f16sr": (2, 4),
         "bf16sr": (2, 4), "f16gsr": (2, 4)}
FLOPS_NODE = 350  # macroscopic update, TRT + Smagorinsky + Guo on f, BGK on g


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: the smoke run's cavity, FP64 (latency and launches)
        dict(name="uniform_f64_16x40", kind="uniform", precision="f64", nx=16, ny=40, ra=1e5, cs=0.1, nu=0.0,
             alpha_mult=1.0, dynamic=False, steps=500),
        # the driver's default run: 64 x 256, Ra = 1e6, FP64
        dict(name="uniform_f64_64x256", kind="uniform", precision="f64", nx=64, ny=256, ra=1e6, cs=0.1, nu=0.0,
             alpha_mult=1.0, dynamic=False, steps=2000),
        # the published Ra = 1e8 run's grid and physics (odd height), FP64
        dict(name="uniform_f64_128x511", kind="uniform", precision="f64", nx=128, ny=511, ra=1e8, cs=0.1, nu=0.001,
             alpha_mult=1.2, dynamic=False, steps=2000),
        # the benchmark's cavity in FP32 and in its headline storage format
        dict(name="uniform_f32_128x512", kind="uniform", precision="f32", nx=128, ny=512, ra=1e8, cs=0.1, nu=0.0,
             alpha_mult=1.0, dynamic=False, steps=4000),
        dict(name="uniform_f16sr_128x512", kind="uniform", precision="f16sr", nx=128, ny=512, ra=1e8, cs=0.1, nu=0.0,
             alpha_mult=1.0, dynamic=False, steps=4000),
        # a large single cavity
        dict(name="uniform_f16sr_512x2048", kind="uniform", precision="f16sr", nx=512, ny=2048, ra=1e8, cs=0.1,
             nu=0.0, alpha_mult=1.0, dynamic=False, steps=4000),
        # the dynamic subgrid model (--dynamic-smag) on the default grid
        dict(name="dynamic_f64_64x256", kind="uniform", precision="f64", nx=64, ny=256, ra=1e7, cs=0.1, nu=0.0,
             alpha_mult=1.0, dynamic=True, steps=500),
        # the 64-cavity sweep, plain and in 16-bit storage
        dict(name="batch_f32_64", kind="batch", precision="f32", cavities=64, first=0, width=0, steps=2000),
        dict(name="batch_f16sr_64", kind="batch", precision="f16sr", cavities=64, first=0, width=0, steps=3000),
        # the gradient run: 96 x 384, Ra = 1e7, a checkpoint every 500 steps
        dict(name="adjoint_f32_96x384", kind="adjoint", precision="f32", nx=96, ny=384, ra=1e7, steps=20000,
             checkpoint=500),
        # the block-refined driver's default (2 levels, FP64)
        dict(name="octree_f64_64x256_l2", kind="octree", precision="f64", nx=64, ny=256, bl=8, levels=2, ra=1e6,
             dynamic=False, steps=512),
        # the large block-refined run: FP32 with binary16 fine levels
        dict(name="octree_f32f16_256x1024_l3", kind="octree", precision="f32_f16", nx=256, ny=1024, bl=16, levels=3,
             ra=1e8, dynamic=False, steps=512),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _ra(rng, ny):
    """A Rayleigh number that a grid of this height resolves."""
    return float("%.3g" % _log(rng, 1e5, max(2e5, min(1e8, 400.0 * ny * ny))))


def draw(rng):
    kind = rng.choice(("uniform", "uniform", "uniform", "dynamic", "batch", "adjoint", "octree", "octree"))
    if kind in ("uniform", "dynamic"):
        dyn = kind == "dynamic"
        ny = int(_log(rng, 40, 512 if dyn else 2048))
        nx = max(16, min(512, int(ny * rng.uniform(0.22, 0.5))))
        precision = "f64" if dyn else rng.choice(("f64", "f32", "f32", "f16sr", "f16", "bf16sr"))
        steps = int(max(100, min(4000, (3e7 if dyn else 8e8) / (nx * ny))))
        return dict(kind="uniform", precision=precision, nx=nx, ny=ny, ra=_ra(rng, ny),
                    cs=round(rng.uniform(0.08, 0.12), 3), nu=0.0, alpha_mult=1.0, dynamic=dyn, steps=steps)
    if kind == "batch":
        return dict(kind="batch", precision=rng.choice(("f32", "f16sr", "f16", "bf16sr")),
                    cavities=int(_log(rng, 2, 64.99)), first=rng.randrange(3), width=rng.choice((0, -1, 3)),
                    steps=rng.randrange(300, 2000))
    if kind == "adjoint":
        ny = int(_log(rng, 64, 400))
        return dict(kind="adjoint", precision=rng.choice(("f32", "f32", "f64")), nx=max(16, ny // 4), ny=ny,
                    ra=float("%.3g" % _log(rng, 1e5, min(1e7, 100.0 * ny * ny))), steps=rng.randrange(500, 1500),
                    checkpoint=rng.choice((100, 125, 250)))
    levels = rng.choice((2, 3))
    ny = int(_log(rng, 64, 1024))
    nx = max(24, min(256, int(ny * rng.uniform(0.22, 0.4))))
    dyn = rng.random() < 0.25
    return dict(kind="octree", precision="f64" if dyn else rng.choice(("f64", "f32", "f32_f16")), nx=nx, ny=ny,
                bl=max(3, nx // rng.choice((8, 12, 16))), levels=levels, ra=_ra(rng, ny), dynamic=dyn,
                steps=int(max(16, min(512, (1e6 if dyn else 4e7) / (nx * ny)))))


def _batch_sizes(case):
    """Widths and heights of a batch's cavities: the sweep's three grids in turn (`width` added to each width)."""
    grids = [BATCH_GRIDS[(case["first"] + i) % 3] for i in range(case["cavities"])]
    return [(nx + case["width"], ny) for nx, ny in grids]


def _octree_grids(case):
    """(nx, ny) of L0, an L1 block and an L2 strip."""
    l1 = (2 * case["bl"] + 3, 2 * (case["ny"] - 1) + 3)
    return (case["nx"], case["ny"]), l1, (7, 2 * (l1[1] - 3) + 3)


def work(case):
    if case["kind"] == "batch":
        nodes = sum(nx * ny for nx, ny in _batch_sizes(case)) * case["steps"]
    elif case["kind"] == "octree":
        l0, l1, l2 = (nx * ny for nx, ny in _octree_grids(case))
        # every level twice per step of the coarser one, L2 in the first L1 sub-step only
        fine = 4 * l1 + (4 * l2 if case["levels"] == 3 else 0)
        pops = {"f64": (8, 8, 8), "f32": (4, 4, 4), "f32_f16": (4, 2, 4)}[case["precision"]]
        per = [36 * pops[0] + 2 * pops[2], 36 * pops[1] + 2 * pops[2]]
        return {"bytes": case["steps"] * (l0 * per[0] + fine * per[1]), "flops": case["steps"] * (l0 + fine) * FLOPS_NODE}
    else:
        nodes = case["nx"] * case["ny"] * case["steps"]
    pop, fy = STORE[case["precision"]]
    if case["kind"] == "adjoint":
        # forward, recomputation (its states kept), and the reverse step: the state and the adjoints read, the adjoints written
        return {"bytes": nodes * (2 * (36 * pop + 2 * fy) + 18 * pop + fy + 2 * 19 * fy), "flops": nodes * 5 * FLOPS_NODE}
    # the dynamic model's box filters, tensors and coefficients: about twice the collision again
    return {"bytes": nodes * (36 * pop + 2 * fy), "flops": nodes * FLOPS_NODE * (3 if case.get("dynamic") else 1)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _fields(nx, ny, seed, shape=()):
    """A smooth convection cell with noise: velocities of the calibrated size, theta stratified between the walls."""
    rng = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, nx)[None, :]
    y = np.linspace(0.0, 1.0, ny)[:, None]
    a = UTARGET * (0.3 + 0.4 * rng.random())
    u = -a * nx / ny * np.sin(np.pi * x) ** 2 * np.sin(2 * np.pi * y)
    v = a * np.sin(2 * np.pi * x) * np.sin(np.pi * y) ** 2
    t = 0.5 - x + 0.2 * np.sin(np.pi * x) * (y - 0.5) + 1e-3 * (2 * rng.random((ny, nx)) - 1)
    rho = 1.0 + 1e-5 * (2 * rng.random((ny, nx)) - 1)
    wall = (x == 0) | (x == 1) | (y == 0) | (y == 1)
    return tuple(np.ascontiguousarray(f, dtype=np.float64).reshape(-1)
                 for f in (rho, np.where(wall, 0.0, u), np.where(wall, 0.0, v), t))


def _profile(ny, seed):
    return 0.5 + 0.01 * (2 * np.random.default_rng(seed + 77).random(ny) - 1)


def _warm_steps(case):
    """Past the spin-up ramp of the viscosity and of the buoyancy."""
    return min(max(case["ny"] // 10, 200), 2000) + 64


def _batch_configs(case, seed):
    rng = np.random.default_rng(seed)
    return [dict(nx=nx, ny=ny, ra=float(10.0 ** rng.uniform(6, 8)), cs=float(rng.uniform(0.08, 0.12)),
                 seed=int(seed) * 1000 + i) for i, (nx, ny) in enumerate(_batch_sizes(case))]


def prepare(case, seed):
    from cfd_cavity_b200 import CavityBatch, CavitySolver
    from cfd_cavity_b200.octree import OctreeSolver

    if case["kind"] == "batch":
        b = CavityBatch(_batch_configs(case, seed), precision=case["precision"])
        b.autotune()
        b.step(_warm_steps(dict(ny=512)))
        b.sync()
        return case, b, None
    if case["kind"] == "octree":
        s = OctreeSolver(case["nx"], case["ny"], case["bl"], case["ra"], PR, UTARGET, int(seed), levels=case["levels"],
                         precision=case["precision"])
        if case["dynamic"]:
            s.set_dynamic_sgs(True)
        s.sync()
        return case, s, None
    fields = _fields(case["nx"], case["ny"], seed)
    if case["kind"] == "adjoint":
        s = CavitySolver(case["nx"], case["ny"], case["ra"], PR, 0.1, PR_T, UTARGET, int(seed),
                         precision=case["precision"], t_hot_profile=_profile(case["ny"], seed))
        return case, s, fields
    s = CavitySolver(case["nx"], case["ny"], case["ra"], PR, case["cs"], PR_T, UTARGET, int(seed),
                     alpha_mult=case["alpha_mult"], nu_override=case["nu"] or None, precision=case["precision"])
    s.init_from_fields(*fields)
    if case["dynamic"]:
        s.set_dynamic_sgs(True)
    else:
        s.step(_warm_steps(case))
    s.sync()
    return case, s, None


def run(state):
    case, s, fields = state
    if case["kind"] == "batch":
        s.step(case["steps"])
        every = [s.fields(i) for i in range(len(s))]
        return {k: np.concatenate([f[k] for f in every]) for k in every[0]}
    if case["kind"] == "octree":
        s.step_cavity(case["steps"])
        out = {"diag": [s.diag()[k] for k in ("nu_hot", "nu_hot_link0", "nu_cold", "nu_hot_fine", "mass")]}
        for lvl in range(3 if case["levels"] == 2 else 5):
            d = s.level(lvl)
            out["level%d" % lvl] = {k: d[k] for k in ("rho", "ux", "uy", "temp")}
        return out
    if case["kind"] == "adjoint":
        s.init_from_fields(*fields)
        n = case["steps"]
        j, grad_theta, grad_cs, _ = s.adjoint_nusselt(n, 2 * n // 3 + 1, case["checkpoint"])
        return {"objective": j, "grad_theta": grad_theta, "grad_cs": grad_cs}
    s.step(case["steps"])
    d = s.diag()
    return {**s.fields(), "diag": [d[k] for k in ("nusselt_hot", "nusselt_cold", "nusselt_hot_wall_link", "total_mass")]}


# ---------------------------------------------------------------------------
# The reference's time step in 64 bits (src/uniform/solver.rs, src/octree/)
# ---------------------------------------------------------------------------
_CX = (0, 1, 0, 1, -1, -1, 0, -1, 1)
_CY = (0, 0, 1, 1, 1, 0, -1, -1, -1)
_OPP = [0, 5, 6, 7, 8, 1, 2, 3, 4]
_W = (4 / 9, 1 / 9, 1 / 9, 1 / 36, 1 / 36, 1 / 9, 1 / 9, 1 / 36, 1 / 36)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device=_device())


def _dirs(ref):
    """c_x, c_y and w, shaped to go with populations (9, ...)."""
    shape = (9,) + (1,) * (ref.dim() - 1)
    return (torch.tensor(v, dtype=torch.float64, device=ref.device).reshape(shape) for v in (_CX, _CY, _W))


def _eq(a, u, v, ndim_like):
    cx, cy, w = _dirs(ndim_like)
    eu = cx * u + cy * v
    return w * a * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u + v * v))


def _collide(f, g, rho, u, v, t, beta, nu, alpha, nut=None, at=None, cs=0.0, tau_s=1.0, pr_t=PR_T):
    """TRT (Lambda = 3/16) with the Guo force for f, BGK for g; nu_t from pi_neq unless given."""
    cx, cy, w = _dirs(f)
    df = f - _eq(rho, u, v, f)
    if nut is None:
        pxx, pxy, pyy = ((df * c).sum(0) for c in (cx * cx, cx * cy, cy * cy))
        nut = cs ** 2 * torch.sqrt(pxx ** 2 + 2 * pxy ** 2 + pyy ** 2) / (2 / 3 * tau_s * rho)
        at = nut / pr_t
    tp = 0.5 + 3 * (nu + nut)
    tm = 0.5 + 3 / 16 / (tp - 0.5)
    fy = rho * beta * t
    s_minus = w * 3 * cy * fy
    s_plus = w * (3 * (cy - v) + 9 * (cx * u + cy * v) * cy) * fy - s_minus
    do = df[_OPP]
    f = f - 0.5 * (df + do) / tp - 0.5 * (df - do) / tm + (1 - 0.5 / tm) * s_minus + (1 - 0.5 / tp) * s_plus
    g = g - (g - _eq(t, u, v, g)) / (0.5 + 3 * (alpha + at))
    return f, g, fy, nut


def _shift(p):
    """Every population from its upwind node, periodic; the callers mend the edges."""
    return torch.stack([torch.roll(p[i], (_CY[i], _CX[i]), (-2, -1)) for i in range(9)])


_masks = {}


def _inside(ny, nx, device):
    """Where each direction's upwind node lies in the grid, (9, ny, nx)."""
    key = (ny, nx, str(device))
    if key not in _masks:
        y, x = torch.meshgrid(torch.arange(ny, device=device), torch.arange(nx, device=device), indexing="ij")
        _masks.clear()
        _masks[key] = torch.stack([(x - _CX[i] >= 0) & (x - _CX[i] < nx) & (y - _CY[i] >= 0) & (y - _CY[i] < ny)
                                   for i in range(9)])
    return _masks[key]


def _moments(f, g, fy):
    cx, cy, _ = _dirs(f)
    rho = f.sum(0)
    return rho, (f * cx).sum(0) / rho, ((f * cy).sum(0) + 0.5 * fy) / rho, g.sum(0)


def _rest(rho):
    """1 inside, 0 on the four walls (no-slip)."""
    m = torch.zeros_like(rho)
    m[..., 1:-1, 1:-1] = 1.0
    return m


class _Uniform:
    """One cavity, or a stack of cavities of one size; scalars may be (n, 1, 1)."""

    def __init__(self, nx, ny, ra, cs, nu=0.0, alpha_mult=1.0, hot=None):
        self.nx, self.ny, self.cs = nx, ny, cs
        lz = ny - 1.0
        cal = (UTARGET * math.sqrt(PR) * lz / (1.7 * ra ** 0.5)) ** (2 / 3)
        cal = torch.clamp(cal, min=0.002) if torch.is_tensor(cal) else max(cal, 0.002)
        self.nu = nu if nu else cal
        self.alpha = self.nu / PR * alpha_mult
        self.beta = ra * self.nu * (self.nu / PR) / lz ** 3
        self.spin = min(max(ny // 10, 200), 2000)
        self.step_no = 0
        self.hot = _t(np.full(ny, 0.5)) if hot is None else hot
        self.fy = self.nut = None

    def start(self, rho, u, v, t):
        self.rho, self.t = rho, t
        like = torch.zeros((9,) + tuple(t.shape), dtype=torch.float64, device=t.device)
        self.f, self.g = _eq(rho, u, v, like), _eq(t, u, v, like)
        self.u, self.v = u * _rest(u), v * _rest(v)

    def step(self, dynamic=False):
        beta = self.beta * min(1.0, self.step_no / self.spin)
        nu_s = torch.clamp(self.nu, min=0.002 / 3) if torch.is_tensor(self.nu) else max(self.nu, 0.002 / 3)
        nut = at = None
        if dynamic:
            nut, at = _model(self.f, self.rho, self.u, self.v, self.t, 0.5 + 3 * nu_s, self.nu, self.alpha)
        f, g, self.fy, self.nut = _collide(self.f, self.g, self.rho, self.u, self.v, self.t, beta, self.nu, self.alpha,
                                           nut, at, cs=self.cs, tau_s=0.5 + 3 * nu_s)
        ok = _inside(self.ny, self.nx, f.device)
        if f.dim() == 4:
            ok = ok[:, None]
        self.f = torch.where(ok, _shift(f), f[_OPP])
        # isothermal columns, then the adiabatic rows copy their neighbours
        _, _, w = _dirs(f)
        hot = (w[..., 0] * self.hot).unsqueeze(-1).expand(g.shape[:-1] + (1,))
        cold = (w[..., 0] * torch.full_like(self.hot, T_COLD)).unsqueeze(-1).expand(g.shape[:-1] + (1,))
        g = torch.cat([hot, _shift(g)[..., 1:-1], cold], -1)
        self.g = torch.cat([g[..., 1:2, :], g[..., 1:-1, :], g[..., -2:-1, :]], -2)
        self.rho, u, v, self.t = _moments(self.f, self.g, self.fy)
        inside = _rest(self.rho)
        self.u, self.v = u * inside, v * inside
        self.step_no += 1

    def nusselt(self, a, b):
        return (self.t[..., a] - self.t[..., b]).abs().mean(-1) * (self.ny - 1.0)


def _box(p, width=2):
    """The test filter: the mean over `width` nodes each way from the node on (width 2), cut at the walls."""
    s, c = torch.zeros_like(p), torch.zeros_like(p)
    ny, nx = p.shape[-2:]
    for j in range(width):
        for i in range(width):
            s[: ny - j, : nx - i] += p[j:, i:]
            c[: ny - j, : nx - i] += 1
    return s / c


def _grad(p):
    x = torch.cat([p[:, :1], p, p[:, -1:]], 1)
    y = torch.cat([p[:1], p, p[-1:]], 0)
    return 0.5 * (x[:, 2:] - x[:, :-2]), 0.5 * (y[2:] - y[:-2])


def _model(f, rho, u, v, t, tau_s, nu, alpha, a=0.5, nu_min=-0.1, eta=2.0):
    """The dynamic mixed-scale model (src/uniform/solver.rs:562-828): nu_t and alpha_t per node."""
    cx, cy, _ = _dirs(f)
    df = f - _eq(rho, u, v, f)
    pxx, pxy, pyy = ((df * c).sum(0) for c in (cx * cx, cx * cy, cy * cy))
    den = 2 / 3 * tau_s * rho
    shxx, shxy, shyy = -pxx / den, -pxy / den, -pyy / den
    smh = torch.sqrt(pxx ** 2 + 2 * pxy ** 2 + pyy ** 2) / den
    ub, vb, tb = _box(u), _box(v), _box(t)
    (uxx, uxy), (vxx, vxy), (gbx, gby), (gtx, gty) = _grad(ub), _grad(vb), _grad(tb), _grad(t)
    sxx, syy, sxy = uxx, vxy, 0.5 * (vxx + uxy)
    smb = torch.sqrt(sxx ** 2 + 2 * sxy ** 2 + syy ** 2)
    du2 = (u - ub) ** 2 + (v - vb) ** 2
    qsm = torch.sqrt(0.5 * du2) / 2
    phi = 0.5 * (t - tb).abs() * torch.sqrt(0.5 * du2)
    tmh = torch.sqrt(2 * ((gtx * shxx + gty * shxy) ** 2 + (gtx * shxy + gty * shyy) ** 2))
    tmb = torch.sqrt(2 * ((gbx * sxx + gby * sxy) ** 2 + (gbx * sxy + gby * syy) ** 2))
    nt = (eta * eta * smb) ** a * (eta * _box(qsm)) ** (1 - a)
    ng = smh ** a * qsm ** (1 - a)
    kt = (eta ** 3 * tmb) ** a * (eta * _box(phi)) ** (1 - a)
    kg = tmh ** a * phi ** (1 - a)
    mxx, mxy, myy = nt * sxx - ng * shxx, nt * sxy - ng * shxy, nt * syy - ng * shyy
    mx, my = kt * gbx - kg * gtx, kt * gby - kg * gty
    lxx, lxy, lyy = _box(u * u) - ub * ub, _box(u * v) - ub * vb, _box(v * v) - vb * vb
    tr = (lxx + lyy) / 3
    ltx, lty = _box(u * t) - ub * tb, _box(v * t) - vb * tb

    def lilly(num, dn):
        num, dn = _box(num), _box(dn)
        c = torch.where(dn > 0, 0.5 * num / torch.where(dn > 0, dn, torch.ones_like(dn)), torch.zeros_like(dn))
        return torch.nan_to_num(c, nan=0.0, posinf=0.0, neginf=0.0).clamp(0.0, 0.04)

    cn = lilly((lxx - tr) * mxx + 2 * lxy * mxy + (lyy - tr) * myy, mxx ** 2 + 2 * mxy ** 2 + myy ** 2)
    ck = lilly(ltx * mx + lty * my, mx ** 2 + my ** 2)
    floor = 0.005 / 3
    return (cn * ng).clamp(min=max(nu_min * nu, floor - nu)), (ck * kg).clamp(min=max(nu_min * alpha, floor - alpha))


def _noise(seeds, n):
    """n draws in [0, 1) of xorshift64* (src/uniform/rng.rs) for every seed, (len(seeds), n)."""
    s = np.array([k | 1 for k in seeds], dtype=np.uint64)
    out = np.empty((n, len(seeds)))
    with np.errstate(over="ignore"):
        for i in range(n):
            s ^= s >> np.uint64(12)
            s ^= s << np.uint64(25)
            s ^= s >> np.uint64(27)
            out[i] = (s * np.uint64(0x2545F4914F6CDD1D)) >> np.uint64(11)
    return out.T / 2.0 ** 53


def _exact_uniform(case, seed):
    nx, ny = case["nx"], case["ny"]
    m = _Uniform(nx, ny, case["ra"], case["cs"], case["nu"], case["alpha_mult"])
    m.start(*(_t(f).reshape(ny, nx) for f in _fields(nx, ny, seed)))
    for _ in range((0 if case["dynamic"] else _warm_steps(case)) + case["steps"]):
        m.step(case["dynamic"])
    out = {k: p.reshape(-1).cpu().numpy() for k, p in (("rho", m.rho), ("ux", m.u), ("uy", m.v), ("temperature", m.t),
                                                       ("nu_t", m.nut), ("fy_node", m.fy))}
    out["diag"] = [float(x) for x in (m.nusselt(1, 2), m.nusselt(-2, -3), m.nusselt(0, 1), m.rho.sum())]
    return out


def _exact_batch(case, seed):
    cfg = _batch_configs(case, seed)
    out = [None] * len(cfg)
    for nx, ny in sorted({(c["nx"], c["ny"]) for c in cfg}):
        at = [i for i, c in enumerate(cfg) if (c["nx"], c["ny"]) == (nx, ny)]
        col = lambda key: _t([cfg[i][key] for i in at]).reshape(-1, 1, 1)  # noqa: E731
        t = _t(1e-4 * (2 * _noise([cfg[i]["seed"] for i in at], nx * ny) - 1)).reshape(len(at), ny, nx)
        m = _Uniform(nx, ny, col("ra"), col("cs"))
        m.start(torch.ones_like(t), torch.zeros_like(t), torch.zeros_like(t), t)
        for _ in range(_warm_steps(dict(ny=512)) + case["steps"]):
            m.step()
        for j, i in enumerate(at):
            out[i] = {k: p[j].reshape(-1).cpu().numpy() for k, p in
                      (("rho", m.rho), ("ux", m.u), ("uy", m.v), ("temperature", m.t), ("nu_t", m.nut),
                       ("fy_node", m.fy))}
    return {k: np.concatenate([o[k] for o in out]) for k in out[0]}


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    nx, ny, n = case["nx"], case["ny"], case["steps"]
    hot = _t(_profile(ny, seed)).requires_grad_(True)
    cs = _t(0.1).requires_grad_(True)
    first = 2 * n // 3 + 1
    rows = torch.arange(ny, device=hot.device).clamp(1, ny - 2)
    start = [_t(f).reshape(ny, nx) for f in _fields(nx, ny, seed)]
    m = _Uniform(nx, ny, case["ra"], cs)
    m.start(*start)

    def stretch(k0, k1, f, g, rho, u, v, t, hot, cs):
        m.hot, m.cs, m.step_no = hot[rows], cs, k0
        m.f, m.g, m.rho, m.u, m.v, m.t = f, g, rho, u, v, t
        j = torch.zeros((), dtype=torch.float64, device=f.device)
        for k in range(k0, k1):
            m.step()
            if k + 1 >= first:
                j = j + m.nusselt(1, 2)
        return m.f, m.g, m.rho, m.u, m.v, m.t, j

    state, total = (m.f, m.g, m.rho, m.u, m.v, m.t), 0.0
    for k in range(0, n, 25):
        *state, j = checkpoint(stretch, k, min(k + 25, n), *state, hot, cs, use_reentrant=False)
        total = total + j
    total = total / (n - first + 1)
    total.backward()
    return {"objective": float(total.detach()), "grad_theta": hot.grad.cpu().numpy(), "grad_cs": float(cs.grad)}


class _Level:
    def __init__(self, nx, ny, t, hot, cold, block):
        self.nx, self.ny, self.hot, self.cold, self.block = nx, ny, hot, cold, block
        t = _t(t).reshape(ny, nx)
        z = torch.zeros_like(t)
        self.rho, self.u, self.v, self.t, self.fy = torch.ones_like(t), z, z, t, z
        like = torch.zeros((9, ny, nx), dtype=torch.float64, device=t.device)
        self.f, self.g = _eq(self.rho, z, z, like), _eq(t, z, z, like)
        self.nut = self.at = z
        lo = 1 if block else 0
        inner = torch.zeros((ny, nx), dtype=torch.bool, device=t.device)
        inner[lo: ny - lo, lo: nx - lo] = True
        y, x = torch.meshgrid(torch.arange(ny, device=t.device), torch.arange(nx, device=t.device), indexing="ij")
        src = [(x - _CX[i], y - _CY[i]) for i in range(9)]
        if block:
            bounce = [((sx == 0) & hot) | ((sx == nx - 1) & cold) | (sy == 0) | (sy == ny - 1) for sx, sy in src]
        else:
            bounce = [(sx < 0) | (sx >= nx) | (sy < 0) | (sy >= ny) for sx, sy in src]
        self.inner, self.bounce = inner, torch.stack(bounce)
        wall = torch.zeros_like(inner)
        wall[lo] = wall[ny - 1 - lo] = True
        if hot:
            wall[:, lo] = True
        if cold:
            wall[:, nx - 1 - lo] = True
        self.wall = wall

    def model(self, nu, alpha):
        self.nut, self.at = _model(self.f, self.rho, self.u, self.v, self.t, 0.5 + 3 * nu, nu, alpha)

    def step(self, nu, alpha, beta, dynamic):
        zero = torch.zeros_like(self.rho)
        f, g, fy, _ = _collide(self.f, self.g, self.rho, self.u, self.v, self.t, beta, nu, alpha,
                               self.nut if dynamic else zero, self.at if dynamic else zero)
        f, g = (torch.where(self.inner, a, b) for a, b in ((f, self.f), (g, self.g)))
        self.fy = torch.where(self.inner, fy, self.fy)
        fs = torch.where(self.bounce, f[_OPP], _shift(f))
        gs = torch.where(self.bounce, g, _shift(g))
        self.f, g = torch.where(self.inner, fs, f), torch.where(self.inner, gs, g)
        _, _, w = _dirs(f)
        lo, nx, ny = (1 if self.block else 0), self.nx, self.ny
        if self.hot:
            g[:, :, lo] = w[..., 0] * 0.5
        if self.cold:
            g[:, :, nx - 1 - lo] = w[..., 0] * T_COLD
        if self.block:
            g[:, 1, 1:-1], g[:, ny - 2, 1:-1] = g[:, 2, 1:-1].clone(), g[:, ny - 3, 1:-1].clone()
            g[:, :, 0], g[:, :, nx - 1] = g[:, :, 1].clone(), g[:, :, nx - 2].clone()
        g[:, 0], g[:, ny - 1] = g[:, 1].clone(), g[:, ny - 2].clone()
        self.g = g
        self.rho, u, v, self.t = _moments(self.f, g, self.fy)
        self.u, self.v = u.masked_fill(self.wall, 0.0), v.masked_fill(self.wall, 0.0)

    def neq(self):
        return torch.cat([torch.stack([self.rho, self.u, self.v, self.t]), self.f - _eq(self.rho, self.u, self.v, self.f),
                          self.g - _eq(self.t, self.u, self.v, self.g)]).reshape(22, -1)

    def put(self, k, mean, even, odd, th):
        """Populations at nodes k from interpolated moments and rescaled non-equilibrium parts; their moments."""
        rho, u, v, t = mean[:4]
        fn, gn = mean[4:13], mean[13:]
        like = fn
        f = _eq(rho, u, v, like) + even * 0.5 * (fn + fn[_OPP]) + odd * 0.5 * (fn - fn[_OPP])
        g = _eq(t, u, v, like) + th * gn
        cx, cy, _ = _dirs(f)
        for name, p in (("f", f), ("g", g)):
            q = getattr(self, name).reshape(9, -1).clone()
            q[:, k] = p
            setattr(self, name, q.reshape(9, self.ny, self.nx))
        rho = f.sum(0)
        for name, p in (("rho", rho), ("u", (f * cx).sum(0) / rho), ("v", (f * cy).sum(0) / rho), ("t", g.sum(0))):
            q = getattr(self, name).reshape(-1).clone()
            q[k] = p
            setattr(self, name, q.reshape(self.ny, self.nx))


def _bilinear(x, y, nx, ny):
    ix, iy = np.clip(np.floor(x).astype(np.int64), 0, nx - 2), np.clip(np.floor(y).astype(np.int64), 0, ny - 2)
    fx, fy = x - ix, y - iy
    k = iy * nx + ix
    return np.stack([k, k + 1, k + nx, k + nx + 1]), np.stack([(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy])


class _Link:
    """A coarse level and a block on it: the ghost ring's stencils and the coincident nodes (src/octree/grid.rs)."""

    def __init__(self, c, f, bx, by, skip_left=False, skip_bottom=False):
        self.c, self.f = c, f
        b, a = (m.reshape(-1) for m in np.meshgrid(np.arange(f.ny), np.arange(f.nx), indexing="ij"))
        ring = (a == 0) | (b == 0) | (a == f.nx - 1) | (b == f.ny - 1)
        kc, w = _bilinear(bx - 0.5 + 0.5 * a[ring], by - 0.5 + 0.5 * b[ring], c.nx, c.ny)
        dev = c.t.device
        self.ghost = torch.as_tensor((b * f.nx + a)[ring], device=dev)
        self.kc, self.w = torch.as_tensor(kc, device=dev), _t(w)
        x1, y1 = bx + (f.nx - 3) // 2, by + (f.ny - 3) // 2
        cy, cx = (m.reshape(-1) for m in np.meshgrid(np.arange(by, y1), np.arange(bx, x1), indexing="ij"))
        keep = (cx > 0) & (cx + 1 < c.nx) & (cy > 0) & (cy + 1 < c.ny)
        keep &= ~((skip_left & (cx == bx)) | (skip_bottom & (cy == by)))
        cx, cy = cx[keep], cy[keep]
        self.coin = torch.as_tensor(cy * c.nx + cx, device=dev)
        fa, fb = 2 * (cx - bx) + 1, 2 * (cy - by) + 1
        ww = (0.25, 0.5, 0.25)
        self.kf = torch.as_tensor(np.stack([(fb + j - 1) * f.nx + fa + i - 1 for j in range(3) for i in range(3)]), device=dev)
        self.wf = _t([ww[i] * ww[j] for j in range(3) for i in range(3)])

    def down(self, xi):
        n = self.c.neq()
        self.f.put(self.ghost, sum(self.w[s] * n[:, self.kc[s]] for s in range(4)), *xi)

    def up(self, xi):
        n = self.f.neq()
        self.c.put(self.coin, sum(self.wf[s] * n[:, self.kf[s]] for s in range(9)), *(1 / x for x in xi))


def _exact_octree(case, seed):
    nx, ny, bl, levels, dyn = case["nx"], case["ny"], case["bl"], case["levels"], case["dynamic"]
    (_, _), (nx1, ny1), (nx2, ny2) = _octree_grids(case)
    lz = ny - 1.0
    nu = max((UTARGET * math.sqrt(PR) * lz / (1.7 * math.sqrt(case["ra"]))) ** (2 / 3), 0.002)
    al = nu / PR
    beta = case["ra"] * nu * al / lz ** 3
    t0 = 0.5 - np.arange(nx)[None, :] / (nx - 1.0) + 1e-3 * (2 * _noise([int(seed)], nx * ny).reshape(ny, nx) - 1)
    t0 = t0.reshape(-1)

    def fine(x, y, w, h):
        k, wt = _bilinear(np.tile(x, h), np.repeat(y, w), nx, ny)
        return (wt * t0[k]).sum(0)

    l0 = _Level(nx, ny, t0, True, True, False)
    bx = (0, nx - 1 - bl)
    l1, l2, a, b = [], [], [], []
    for s in range(2):
        x1, y1 = bx[s] - 0.5 + 0.5 * np.arange(nx1), -0.5 + 0.5 * np.arange(ny1)
        l1.append(_Level(nx1, ny1, fine(x1, y1, nx1, ny1), s == 0, s == 1, True))
        a.append(_Link(l0, l1[s], bx[s], 0))
        if levels == 3:
            sx = 1 if s == 0 else nx1 - 4
            x2 = bx[s] - 0.5 + 0.5 * (sx - 0.5 + 0.5 * np.arange(nx2))
            y2 = -0.5 + 0.5 * (1 - 0.5 + 0.5 * np.arange(ny2))
            l2.append(_Level(nx2, ny2, fine(x2, y2, nx2, ny2), s == 0, s == 1, True))
            b.append(_Link(l1[s], l2[s], sx, 1, skip_left=True, skip_bottom=True))

    def xi(k, cn, ca, fn, fa):
        """Rescaling factors between levels k and k + 1 with mean nu_t / alpha_t of each."""
        c, f = 2 ** k, 2 ** (k + 1)
        return (0.5 * (0.5 + 3 * (f * nu + fn)) / (0.5 + 3 * (c * nu + cn)), 0.5,
                0.5 * (0.5 + 3 * (f * al + fa)) / (0.5 + 3 * (c * al + ca)))

    for _ in range(case["steps"]):
        if dyn:
            l0.model(nu, al)
        means = [float(sum(getattr(p, q).mean() for p in l1) / 2) for q in ("nut", "at")]
        xa = xi(0, float(l0.nut.mean()), float(l0.at.mean()), *means)
        l0.step(nu, al, beta, dyn)
        for s in range(2):
            a[s].down(xa)
        for s in range(2):
            if dyn:
                l1[s].model(2 * nu, 2 * al)
            l1[s].step(2 * nu, 2 * al, 0.5 * beta, dyn)
            if levels == 3:
                xb = xi(1, *(float(getattr(p[s], q).mean()) for p in (l1, l2) for q in ("nut", "at")))
                b[s].down(xb)
                for _ in range(2):
                    if dyn:
                        l2[s].model(4 * nu, 4 * al)
                    l2[s].step(4 * nu, 4 * al, 0.25 * beta, dyn)
                b[s].up(xb)
            if dyn:
                l1[s].model(2 * nu, 2 * al)
            l1[s].step(2 * nu, 2 * al, 0.5 * beta, dyn)
        for s in range(2):
            a[s].up(xa)
    hot = [float((l0.t[:, i] - l0.t[:, j]).abs().mean()) * (nx - 1.0) for i, j in ((1, 2), (0, 1), (-2, -3))]
    first = float((l1[0].t[1:-1, 1] - l1[0].t[1:-1, 2]).abs().mean()) * 2 * (nx - 1.0)
    out = {"diag": hot + [first, float(l0.rho.mean())]}
    for i, p in enumerate([l0] + l1 + l2):
        out["level%d" % i] = {k: q.reshape(-1).cpu().numpy() for k, q in
                              (("rho", p.rho), ("ux", p.u), ("uy", p.v), ("temp", p.t))}
    return out


def exact(case, seed):
    # about 0.6 ms a step for the smallest grids, then by the values streamed
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed) if case["steps"] <= 1500 else None
    if case["kind"] == "octree":
        return _exact_octree(case, seed) if case["steps"] * (40 if case["dynamic"] else 12) <= 9000 else None
    if case["kind"] == "batch":
        nodes = sum(nx * ny for nx, ny in _batch_sizes(case))
        return _exact_batch(case, seed) if nodes * case["steps"] <= 2.0e9 else None
    return _exact_uniform(case, seed) if case["nx"] * case["ny"] * case["steps"] <= 2.0e9 else None
