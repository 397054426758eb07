"""The work a user of this framework has it do, as timed cases.

Each case is one whole solve through the public Python entry points: initial cells in host memory
go in, the solver takes its steps, the final cells come back.  `static` cases are the
reference-named calls (FP64, the default of every one of them); `grid` cases hold a device-resident
grid and page-locked buffers, as long runs and FP32 runs do; `batch`, `amr` and `adjoint` are the
many-grid launch, the adaptive driver and the gradient of a solve.

Grids with FP32 storage return their cells rounded to 32 bits, the precision they hold.

`exact` restates the schemes (SLIC and FORCE sweeps, the relativistic primitive recovery, the
Kerr-Schild source step, Level-1 refinement) in plain torch at 64 bits.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import cosmos_gb300 as cg

SUPERBEE, VANLEER, MINBEE = 0, 1, 2
SYSTEM = {"newton": cg.NEWTONIAN, "sr": cg.SR, "gr": cg.GR}
GAMMA = {"newton": 1.4, "sr": 5.0 / 3.0, "gr": 5.0 / 3.0}
# the accretion problem: a unit-mass hole in the middle of a box of 20 masses
GR_BOX = 20.0
GR_HOLE = (1.0, 0.0, 10.0, 10.0, 0.0)


def _case(name, kind, system, ny, nx, precision, steps, order=2, limiter=VANLEER, periodic=False, data="riemann", **more):
    c = dict({"kind": kind, "system": system, "ny": ny, "nx": nx, "precision": precision, "steps": steps,
              "order": order, "limiter": limiter, "periodic": periodic, "data": data}, **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the first run of anybody who switches from the reference: the Sod tube to its final time,
        # one static call, a few cells per step (launches and latency)
        _case("sod 1000 fp64", "static", "newton", 0, 1000, 64, -1, data="sod", t_final=0.25),
        # the reference's 2D Riemann problems by the default (reference-exact) path, odd sizes
        _case("riemann 389x509 fp64", "static", "newton", 389, 509, 64, 40),
        # the same system by the first-order solver, on the small grids of its tests
        _case("riemann 200x200 force fp64", "static", "newton", 200, 200, 64, 60, order=1),
        # a small FP32 grid: many short steps on a grid that stays in cache, SuperBee, ragged edges
        _case("riemann 193x257 fp32", "grid", "newton", 193, 257, 32, 400, limiter=SUPERBEE),
        # the headline grid of the benchmark: production runs in FP32, periodic
        _case("riemann 4096x4096 fp32", "grid", "newton", 4096, 4096, 32, 192, limiter=MINBEE, periodic=True),
        # relativistic shear layers at the benchmark's size, FP32
        _case("shear 2048x2048 sr fp32", "grid", "sr", 2048, 2048, 32, 48, limiter=MINBEE, periodic=True, data="shear"),
        # relativistic Riemann problem by the default path
        _case("riemann 181x230 sr fp64", "static", "sr", 181, 230, 64, 16),
        # accretion onto a hole at the benchmark's size, FP32, one source step on each side
        _case("accretion 1024x1024 gr fp32", "grid", "gr", 1024, 1024, 32, 6, data="accretion"),
        # the same by the default path on a small grid
        _case("accretion 150x150 gr fp64", "static", "gr", 150, 150, 64, 6, data="accretion"),
        # a parameter study: many uneven 1D and 2D grids in one launch
        _case("batch of 48 fp32", "batch", "newton", 0, 0, 32, 40, limiter=MINBEE, grids=48),
        # the reference's adaptive test layout (a cylindrical explosion), default precision
        _case("amr 128x128 fp64", "amr", "newton", 128, 128, 64, -1, data="explosion", t_final=0.1, tol=20.0),
        # fitting an initial state: gradient of a density mismatch through a solve
        _case("adjoint 1024x1024 fp32", "adjoint", "newton", 1024, 1024, 32, 30, limiter=MINBEE, data="smooth"),
    ]


def _data(system, periodic):
    return "accretion" if system == "gr" else "shear" if system == "sr" and periodic else "riemann"


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def steps_for(cells, rate, most):  # a pass of about 0.15 s at most
        return max(4, min(most, int(0.15 * rate / cells)))

    kind = rng.choice(["static", "static", "grid", "grid", "batch", "amr", "adjoint"])
    limiter = rng.choice([SUPERBEE, VANLEER, MINBEE])
    periodic = rng.random() < 0.4
    if kind == "static":
        system = rng.choice(["newton", "newton", "sr", "gr"])
        if system == "newton" and rng.random() < 0.4:
            return _case("", kind, system, 0, size(100, 4000), 64, rng.randint(100, 500), rng.choice([1, 2]), limiter,
                         periodic)  # 1D: a shock tube
        ny, nx = (size(60, 500), size(60, 500)) if system != "gr" else (size(60, 200),) * 2
        rate = {"newton": 1.2e8, "sr": 2e7, "gr": 2e6}[system]
        return _case("", kind, system, ny, nx, 64, steps_for(ny * nx, rate, 80 if system != "gr" else 8),
                     rng.choice([1, 2, 2]) if system != "gr" else 2, limiter if system == "newton" else MINBEE,
                     periodic and system != "gr", _data(system, periodic))
    if kind == "grid":
        system = rng.choice(["newton", "newton", "newton", "sr", "gr"])
        if system == "gr":
            n = size(200, 1024)
            return _case("", kind, system, n, n, 32, 6, data="accretion")
        lo, hi = (100, 4000) if system == "newton" else (100, 2000)
        ny, nx = size(lo, hi), size(lo, hi)
        rate = {"newton": 1.5e10, "sr": 2e9}[system]
        return _case("", kind, system, ny, nx, 32, steps_for(ny * nx, rate, 400), 2,
                     limiter if system == "newton" else MINBEE, periodic, _data(system, periodic))
    if kind == "batch":
        return _case("", kind, "newton", 0, 0, 32, rng.randint(20, 40), 2, limiter, periodic,
                     grids=rng.randint(8, 48))
    if kind == "amr":
        return _case("", kind, "newton", size(40, 128), size(40, 128), 64, -1, rng.choice([1, 2]),
                     data="explosion", t_final=0.03, tol=float(rng.randint(10, 30)))
    ny, nx = size(100, 1000), size(100, 1000)
    return _case("", kind, "newton", ny, nx, 32, rng.randint(10, 30), 2, MINBEE, periodic, "smooth")


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dx(case):
    return GR_BOX / case["nx"] if case["system"] == "gr" else 1.0 / max(case["nx"], 1)


def _quadrants(ny, nx, g, system):
    """Two (1D) or four (2D) constant states with a slight wave on density and pressure."""
    dev = _device()
    q = torch.rand((4, 5), generator=g, dtype=torch.float64)
    lo = torch.tensor([0.4, -0.6, -0.6, 0.0, 0.3] if system == "newton" else [0.6, -0.3, -0.3, 0.0, 0.6])
    hi = torch.tensor([1.5, 0.6, 0.6, 0.0, 1.5] if system == "newton" else [1.4, 0.3, 0.3, 0.0, 1.4])
    q = (lo + (hi - lo) * q).to(dev)
    ph = (2.0 * math.pi * torch.rand(4, generator=g, dtype=torch.float64)).to(dev)
    rows, cols = max(ny, 1), nx
    p = torch.empty((rows, cols, 5), dtype=torch.float64, device=dev)
    hx, hy = cols // 2, rows // 2
    if ny == 0:
        p[:, :hx], p[:, hx:] = q[0], q[1]
        p[..., 2] = 0.0
    else:
        p[:hy, :hx], p[:hy, hx:], p[hy:, :hx], p[hy:, hx:] = q[0], q[1], q[2], q[3]
    x = 2.0 * math.pi * (torch.arange(cols, device=dev, dtype=torch.float64) + 0.5) / cols
    y = 2.0 * math.pi * (torch.arange(rows, device=dev, dtype=torch.float64) + 0.5) / rows
    p[..., 0] *= 1.0 + 0.02 * torch.sin(2.0 * x + ph[0]) * torch.cos(3.0 * y[:, None] + ph[1])
    p[..., 4] *= 1.0 + 0.02 * torch.cos(3.0 * x + ph[2]) * torch.sin(2.0 * y[:, None] + ph[3])
    return p


def _shear(ny, nx, g):
    """A band 0.25 < y < 0.75 moving against its surroundings, joined by tanh profiles."""
    dev = _device()
    ph = 2.0 * math.pi * torch.rand(2, generator=g, dtype=torch.float64).to(dev)
    x = (torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) / nx
    y = ((torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) / ny)[:, None]
    s = torch.tanh((y - 0.25) / 0.01) - torch.tanh((y - 0.75) / 0.01) - 1.0
    p = torch.zeros((ny, nx, 5), dtype=torch.float64, device=dev)
    p[..., 0] = 1.5 + 0.5 * s
    p[..., 1] = 0.5 * s
    p[..., 2] = 0.01 * (torch.sin(4.0 * math.pi * x + ph[0]) + 0.5 * torch.sin(6.0 * math.pi * x + ph[1]))
    p[..., 4] = 1.0
    return p


def _accretion(ny, nx, seed):
    """Gas at rest with one per cent density noise around the hole."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    p = torch.zeros((ny, nx, 5), dtype=torch.float64, device=dev)
    p[..., 0] = torch.exp(0.01 * torch.randn((ny, nx), generator=g, dtype=torch.float64, device=dev))
    p[..., 4] = 0.01
    return p


def _smooth(ny, nx, g):
    """Sines of random phase."""
    dev = _device()
    ph = (2.0 * math.pi * torch.rand(6, generator=g, dtype=torch.float64)).to(dev)
    x = 2.0 * math.pi * (torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) / nx
    y = 2.0 * math.pi * ((torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) / ny)[:, None]
    p = torch.empty((ny, nx, 5), dtype=torch.float64, device=dev)
    p[..., 0] = 1.0 + 0.3 * torch.sin(x + ph[0]) * torch.cos(y + ph[1])
    p[..., 1] = 0.3 * torch.sin(x + y + ph[2])
    p[..., 2] = 0.2 * torch.cos(x + ph[3])
    p[..., 3] = 0.05 * torch.sin(y + ph[4])
    p[..., 4] = 1.0 + 0.2 * torch.cos(x + ph[5])
    return p


def _explosion(ny, nx, g):
    """Dense hot gas inside a circle (the reference's adaptive 2D test)."""
    dev = _device()
    v = torch.rand(3, generator=g, dtype=torch.float64).tolist()
    i = torch.arange(ny, device=dev, dtype=torch.float64)[:, None]
    j = torch.arange(nx, device=dev, dtype=torch.float64)
    inside = torch.sqrt((i - 0.5 * ny) ** 2 + (j - 0.5 * nx) ** 2) <= (0.18 + 0.04 * v[0]) * min(ny, nx)
    p = torch.zeros((ny, nx, 5), dtype=torch.float64, device=dev)
    p[..., 0] = torch.where(inside, 1.0 + 0.1 * v[1], 0.125)
    p[..., 4] = torch.where(inside, 1.0 + 0.1 * v[2], 0.1)
    return p


def _cells(case, seed):
    """The initial cells of a case: (ny, nx, 5) primitives, ny = 1 in 1D."""
    g = torch.Generator().manual_seed(seed)
    ny, nx = case["ny"], case["nx"]
    if case["data"] == "smooth":
        return _smooth(ny, nx, g)
    if case["data"] == "accretion":
        return _accretion(ny, nx, seed)
    if case["data"] == "explosion":
        return _explosion(ny, nx, g)
    if case["data"] == "sod":  # Sod's two states, their strength within a few per cent by seed
        v = torch.rand(2, generator=g, dtype=torch.float64).tolist()
        p = torch.zeros((1, nx, 5), dtype=torch.float64, device=_device())
        left = torch.arange(nx, device=_device()) <= 0.5 * nx
        p[..., 0] = torch.where(left, 1.0 + 0.05 * v[0], 0.125)
        p[..., 4] = torch.where(left, 1.0 + 0.05 * v[1], 0.1)
        return p
    if case["data"] == "shear":
        return _shear(ny, nx, g)
    return _quadrants(ny, nx, g, case["system"])


def _target(case, seed):
    """The density to match: another state of the same kind."""
    return _smooth(case["ny"], case["nx"], torch.Generator().manual_seed(seed + 1))[..., 0].contiguous()


def _batch_shapes(case, seed):
    """Half 1D, half 2D grids, every side log-uniform in [128, 1024]."""
    rng = np.random.default_rng([case["grids"], case["steps"]])  # the study's grids; the seed changes its states
    side = lambda: int(round(float(np.exp(rng.uniform(np.log(128), np.log(1024))))))  # noqa: E731
    return [(side(),) if k % 2 else (side(), side()) for k in range(case["grids"])]


def _batch_cells(case, seed):
    out = []
    for k, sh in enumerate(_batch_shapes(case, seed)):
        g = torch.Generator().manual_seed(seed * 1000 + k)
        out.append(_quadrants(sh[0] if len(sh) == 2 else 0, sh[-1], g, "newton"))
    return out


def _pinned(t):
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return h


def _host(case, t):
    a = t.cpu().numpy()
    return a[0].copy() if case["ny"] == 0 else a


def prepare(case, seed):
    s = {"case": case, "gas": cg.EulerMaterialParameters(GAMMA[case["system"]]), "dx": _dx(case)}
    bc = cg.BC_PERIODIC if case["periodic"] else cg.BC_TRANSMISSIVE
    prec = cg.FP32 if case["precision"] == 32 else cg.FP64
    if case["system"] == "gr":
        s["hole"] = cg.BlackHoleSpacetime(*GR_HOLE)
    if case["kind"] == "batch":
        cells = _batch_cells(case, seed)
        shapes = _batch_shapes(case, seed)
        s["cells"] = [_pinned(c.reshape(sh + (5,))) for c, sh in zip(cells, shapes)]
        s["out"] = [torch.empty(sh + (5,), dtype=torch.float64, pin_memory=True) for sh in shapes]
        s["kept"] = [torch.empty(sh + (5,), dtype=torch.float32) for sh in shapes]
        s["batch"] = cg.Batch(shapes, [1.0 / sh[-1] for sh in shapes], 1.4, prec, bc)
        return s
    cells = _cells(case, seed)
    if case["kind"] in ("static", "amr"):
        s["cells"], s["bc"] = _host(case, cells), bc
        return s
    s["cells"] = _pinned(cells)
    if case["kind"] == "adjoint":
        s["target"] = _target(case, seed).cpu().numpy()
    else:
        s["out"] = torch.empty(cells.shape, dtype=torch.float64, pin_memory=True)
        s["kept"] = torch.empty(cells.shape, dtype=torch.float32)
    s["grid"] = cg.Grid(SYSTEM[case["system"]], tuple(cells.shape[:2]), s["dx"], GAMMA[case["system"]], prec, bc,
                        s.get("hole"))
    return s


# ------------------------------------------------------------------ one pass
CFL = 0.9
FOREVER = 1e30


def run(s):
    c = s["case"]
    steps, t_final = c["steps"], c.get("t_final", FOREVER)
    if c["kind"] == "static":
        if c["system"] == "gr":
            return cg.BlackHoleEulerSecondOrderSolver.solve2D(s["cells"], s["dx"], CFL, t_final, 0.0, c["limiter"], 1,
                                                              s["gas"], s["hole"], max_steps=steps)
        second, first = {"newton": (cg.EulerSecondOrderSolver, cg.EulerFirstOrderSolver),
                         "sr": (cg.RelativisticEulerSecondOrderSolver, cg.RelativisticEulerFirstOrderSolver)}[c["system"]]
        if c["order"] == 1:
            return first.solve(s["cells"], s["dx"], CFL, t_final, s["gas"], boundary=s["bc"], max_steps=steps)
        return second.solve(s["cells"], s["dx"], CFL, t_final, 0.0, c["limiter"], s["gas"], boundary=s["bc"],
                            max_steps=steps)
    if c["kind"] == "amr":
        coarse, fine, cf, ff = cg.EulerAMR.solve2DLevel1AMR(s["cells"], s["dx"], CFL, t_final, c["tol"], c["order"],
                                                            s["gas"])
        return {"coarse": coarse, "fine": fine, "coarse_on": cf, "fine_on": ff}
    if c["kind"] == "batch":
        b = s["batch"]
        for k, cells in enumerate(s["cells"]):
            b.set_prim(k, cells.numpy())
        b.run_begin(CFL, t_final, 0.0, c["limiter"], max_steps=steps)
        b.run_steps(steps)
        b.run_end()
        for k, (out, kept) in enumerate(zip(s["out"], s["kept"])):
            b.get_prim(k, out.numpy())
            kept.copy_(out)
        return s["kept"]
    g = s["grid"]
    g.set_prim(s["cells"].numpy())
    if c["kind"] == "adjoint":
        loss, grad, dts, _ = g.adjoint(s["target"], steps, CFL, 0.0, c["limiter"])
        return {"loss": loss, "grad": torch.from_numpy(grad).float(), "dts": torch.from_numpy(dts).float()}
    g.run_begin(c["order"], CFL, t_final, 0.0, c["limiter"], max_steps=steps)
    g.run_steps(steps)
    g.run_end()
    g.get_prim(s["out"].numpy())
    return s["kept"].copy_(s["out"])


# ------------------------------------------------------------------ what a pass cannot do without
# Arithmetic operations per cell (a division or root counts one): a SLIC sweep is 5 slopes, 5 flux
# evaluations and the conversions between them; the relativistic ones add a recovery of about 150
# operations at every flux; the source step is four source terms and nine fractional evolutions.
SWEEP_FLOPS = {"newton": {2: 300, 1: 130}, "sr": {2: 1100, 1: 700}, "gr": {2: 1500, 1: 900}}
SOURCE_FLOPS = 6000
ADJOINT_FLOPS = 600


def work(case):
    def of(cells, dims, steps, order=case["order"], system=case["system"]):
        per = SWEEP_FLOPS[system][order] * (3 if dims == 2 else 1) + (2 * SOURCE_FLOPS if system == "gr" else 0)
        return cells * steps * per

    host = 80  # bytes of a cell in and out (five doubles each way)
    if case["kind"] == "batch":
        shapes = _batch_shapes(case, 0)
        return {"bytes": sum(int(np.prod(s)) for s in shapes) * host,
                "flops": sum(of(int(np.prod(s)), len(s), case["steps"]) for s in shapes)}
    dims = 2 if case["ny"] else 1
    cells = case["nx"] * max(case["ny"], 1)
    steps = case["steps"] if case["steps"] > 0 else int(case["t_final"] * 2.5 / CFL / _dx(case))
    if case["kind"] == "amr":  # the coarse steps; fine steps run on the refined cells, about a tenth of four times as many
        return {"bytes": cells * (host + 40 * 4), "flops": of(cells, 2, steps) + of(int(0.4 * cells), 2, 2 * steps)}
    if case["kind"] == "adjoint":
        return {"bytes": cells * (host + 8), "flops": of(cells, 2, steps) + cells * steps * 3 * ADJOINT_FLOPS}
    return {"bytes": cells * host, "flops": of(cells, dims, steps)}


# ------------------------------------------------------------------ the schemes in 64 bits
# A state is a tensor (5, lines, cells along the sweep); `at` is the (x, y) of its points.
class Newton:
    coords = False

    def __init__(self, case):
        self.g = GAMMA["newton"]

    def cons(self, p, at):
        r, u, v, w, q = p
        return torch.stack([r, r * u, r * v, r * w, q / (self.g - 1.0) + 0.5 * r * (u * u + v * v + w * w)])

    def prim(self, u, at):
        r = u[0]
        a, b, c = u[1] / r, u[2] / r, u[3] / r
        return torch.stack([r, a, b, c, (self.g - 1.0) * (u[4] - 0.5 * r * (a * a + b * b + c * c))])

    def flux(self, u, axis, at):
        p = self.prim(u, at)
        n = p[1 + axis]
        f = [u[0] * n, u[1] * n, u[2] * n, u[3] * n, (u[4] + p[4]) * n]
        f[1 + axis] = f[1 + axis] + p[4]
        return torch.stack(f)

    def speed(self, p, dims):
        c = torch.sqrt(self.g * p[4] / p[0])
        return p[1].abs() + c if dims == 1 else torch.maximum(p[1].abs(), p[2].abs() + c)


def _recover(D, S, tau, g):
    """Primitives, Lorentz factor and enthalpy from densities: Newton on the quartic to convergence,
    the last step taken differentiably (the implicit-function derivative)."""
    q = (tau + D) ** 2 - (S[0] ** 2 + S[1] ** 2 + S[2] ** 2)
    root = torch.sqrt(q.clamp(min=1e-8))
    dc, ec = D / root, (D + tau) / root
    gm = (g - 1.0) / g
    c0, c1 = -1.0 / g**2, -2.0 * dc * (g - 1.0) / g**2
    c2, c4, eta = (g - 2.0) / g * (ec * ec - 1.0) + 1.0 - (dc * gm) ** 2, ec * ec - 1.0, 2.0 * dc * gm

    def f(x):
        return c4 * x**3 * (x - eta) + c2 * x * x + c1 * x + c0

    def df(x):
        return c1 + 2.0 * c2 * x + 4.0 * c4 * x**3 - 3.0 * eta * c4 * x * x

    with torch.no_grad():
        x = torch.ones_like(dc)
        for _ in range(40):
            step = f(x) / df(x)
            x = x - step
            if not bool((step.abs() > 1e-14).any()):
                break
    if torch.is_grad_enabled():
        x = x - f(x) / df(x).detach()
    W = 0.5 * ec * x * (1.0 + torch.sqrt(1.0 + 4.0 * gm * (1.0 - dc * x) / (ec * x) ** 2))
    h = 1.0 / (dc * x)
    rho = D / W
    rhw = rho * h * W * W
    return rho.clamp(min=1e-8), [s / rhw for s in S], (rhw - D - tau).clamp(min=1e-8), W, h


class Special:
    coords = False

    def __init__(self, case):
        self.g = GAMMA["sr"]

    def cons(self, p, at):
        r, v, q = p[0], p[1:4], p[4]
        W = 1.0 / torch.sqrt(1.0 - (v * v).sum(0))
        m = (r + q * self.g / (self.g - 1.0)) * W * W
        return torch.stack([r * W, m * v[0], m * v[1], m * v[2], m - q - r * W])

    def prim(self, u, at):
        r, v, q, _, _ = _recover(u[0], u[1:4], u[4], self.g)
        return torch.stack([r, *v, q])

    def flux(self, u, axis, at):
        r, v, q, W, h = _recover(u[0], u[1:4], u[4], self.g)
        m, n = r * h * W * W, v[axis]
        f = [r * W * n, m * v[0] * n, m * v[1] * n, m * v[2] * n, (m - r * W) * n]
        f[1 + axis] = f[1 + axis] + q
        return torch.stack(f)

    def speed(self, p, dims):
        c = torch.sqrt(self.g * p[4] / p[0] / (1.0 + p[4] / p[0] * self.g / (self.g - 1.0)))
        return (p[1].abs() if dims == 1 else torch.maximum(p[1].abs(), p[2].abs())) + c


def _inverse(m):
    """Inverse per point; points without one (inside the horizon) get what comes out."""
    one = torch.eye(m.shape[-1], dtype=m.dtype, device=m.device)
    return torch.linalg.inv_ex(torch.where(torch.isfinite(m).all(-1).all(-1)[..., None, None], m, one))[0]


class BlackHole:
    """Kerr-Schild 3+1 form with the reference's conventions (energy with W, one component of its
    null vector as the reference has it)."""
    coords = True

    def __init__(self, case):
        self.g = GAMMA["gr"]
        self.M, self.a, self.bx, self.by, self.bz = GR_HOLE
        self.h = _dx(case)

    def null(self, x, y, z):
        dx, dy, dz = x - self.bx, y - self.by, z - self.bz
        k, n2 = (self.M * self.a) ** 2, dx * dx + dy * dy + dz * dz
        r = torch.sqrt(0.5 * (n2 - k + torch.sqrt((n2 - k) ** 2 + 4.0 * k * dz * dz)))
        H = -self.M * r**3 / (r**4 + k * dz * dz)
        am = self.a * self.M
        l = [-(r * dx + am * dy) / (r * r + k), -(r * dy - am * dx) / (r * r + k), -dz / r + 0.0 * x]
        odd = -((r + dy) - am * dx) / (r * r + k)  # the reference's y component of the 4-vector
        return H, l, odd

    def metric(self, x, y, z=0.0):
        x, y, z = torch.broadcast_tensors(*(torch.as_tensor(v, dtype=torch.float64, device=_device()) for v in (x, y, z)))
        H, l, _ = self.null(x, y, z)
        gam = [[(1.0 if i == j else 0.0) - 2.0 * H * l[i] * l[j] for j in range(3)] for i in range(3)]
        det = (gam[0][0] * (gam[1][1] * gam[2][2] - gam[1][2] * gam[2][1])
               - gam[0][1] * (gam[1][0] * gam[2][2] - gam[1][2] * gam[2][0])
               + gam[0][2] * (gam[1][0] * gam[2][1] - gam[1][1] * gam[2][0]))
        lapse = 1.0 / torch.sqrt(1.0 - 2.0 * H)
        return gam, torch.sqrt(det), lapse, [2.0 * H / (1.0 - 2.0 * H) * v for v in l]

    def excised(self, x, y):
        return torch.sqrt((x - self.bx) ** 2 + (y - self.by) ** 2 + self.bz**2) <= self.M * (1.0 + math.sqrt(1.0 - self.a**2))

    def cons(self, p, at):
        gam, sg, _, _ = self.metric(*at)
        v2 = sum(gam[i][j] * p[1 + i] * p[1 + j] for i in range(3) for j in range(3))
        W = torch.where(v2 > 1.0 - 1e-8, torch.full_like(v2, 1e4), 1.0 / torch.sqrt(1.0 - v2))
        rh = p[0] + p[4] * self.g / (self.g - 1.0)
        return torch.stack([sg * p[0] * W, *(sg * rh * W * W * p[1 + k] for k in range(3)),
                            sg * (rh * W - p[4] - p[0] * W)])

    def prim(self, u, at):
        sg = self.metric(*at)[1]
        r, v, q, _, _ = _recover(u[0] / sg, u[1:4] / sg, u[4] / sg, self.g)
        return torch.stack([r, *v, q])

    def flux(self, u, axis, at):
        _, sg, al, be = self.metric(*at)
        r, v, q, W, h = _recover(u[0] / sg, u[1:4] / sg, u[4] / sg, self.g)
        m, s = r * h * W * W, al * sg
        w = v[axis] - be[axis] / al
        f = [r * W * w, m * v[0] * w, m * v[1] * w, m * v[2] * w, (m - q - r * W) * w + q * v[axis]]
        f[1 + axis] = f[1 + axis] + q
        return s * torch.stack(f)

    def grid_speed(self, p):
        """Largest signed eigenvalue per cell, at the reference's coordinates."""
        ny, nx = p.shape[1:]
        i = torch.arange(ny, device=p.device, dtype=torch.float64)[:, None] / ny
        j = torch.arange(nx, device=p.device, dtype=torch.float64) / nx
        gam, _, al, be = self.metric(i, j)
        m = torch.stack([torch.stack([v.expand(ny, nx) for v in row], -1) for row in gam], -2)
        up = _inverse(m)
        cs = torch.sqrt(self.g * p[4] / p[0] / (1.0 + p[4] / p[0] * self.g / (self.g - 1.0)))
        v = p[1:4]
        v2 = sum(gam[a][b] * v[a] * v[b] for a in range(3) for b in range(3))
        s = torch.zeros_like(cs)
        for k in range(3):
            rt = torch.sqrt((1.0 - v2) * (up[..., k, k] * (1.0 - v2 * cs**2) - v[k] ** 2 * (1.0 - cs**2)))
            pre = al / (1.0 - v2 * cs**2)
            for lam in (al * v[k] - be[k], pre * (v[k] * (1.0 - cs**2) + cs * rt) - be[k],
                        pre * (v[k] * (1.0 - cs**2) - cs * rt) - be[k]):
                s = torch.where(lam > s, lam, s)
        return torch.where(self.excised(j, i), torch.zeros_like(s), s)

    def source_parts(self, x, y):
        """Inverse 4-metric, centred derivatives of lapse, shift and spatial metric, extrinsic
        curvature at the cell centres (the spacetime is static)."""
        x, y = torch.broadcast_tensors(x, y)
        z, h = torch.zeros_like(x), self.h
        H, l, odd = self.null(x, y, z)
        L = [torch.full_like(x, -1.0), l[0], odd, l[2]]
        g4 = torch.stack([torch.stack([(0.0 if i != j else -1.0 if i == 0 else 1.0) - 2.0 * H * L[i] * L[j]
                                       for j in range(4)], -1) for i in range(4)], -2)
        inv = _inverse(g4)
        al = self.metric(x, y)[2]
        da, db, dg, dH, dl = [], [], [], [], []
        for d in range(3):
            hi = [c + (0.5 * h if k == d else 0.0) for k, c in enumerate((x, y, z))]
            lo = [c - (0.5 * h if k == d else 0.0) for k, c in enumerate((x, y, z))]
            (g1, _, a1, b1), (g0, _, a0, b0) = self.metric(*hi), self.metric(*lo)
            (H1, l1, _), (H0, l0, _) = self.null(*hi), self.null(*lo)
            da.append((a1 - a0) / h)
            db.append([(p - q) / h for p, q in zip(b1, b0)])
            dg.append([[(g1[j][k] - g0[j][k]) / h for k in range(3)] for j in range(3)])
            dH.append((H1 - H0) / h)
            dl.append([(p - q) / h for p, q in zip(l1, l0)])
        K = [[al * (-(l[i] * dH[j]) - l[j] * dH[i] - H * dl[j][i] - H * dl[i][j]
                    + sum(2.0 * H * H * (l[i] * l[c] * dl[c][j] + l[j] * l[c] * dl[c][i])
                          + 2.0 * H * l[i] * l[j] * l[c] * dH[c] for c in range(3))) for j in range(3)] for i in range(3)]
        return inv, da, db, dg, K

    def source(self, u, at, parts):
        gam, sg, al, be = self.metric(*at)
        r, v, q, W, h = _recover(u[0] / sg, u[1:4] / sg, u[4] / sg, self.g)
        inv, da, db, dg, K = parts
        ut = W / al
        up = [ut] + [al * ut * v[k] - be[k] * ut for k in range(3)]
        T = [[r * h * up[a] * up[b] + q * inv[..., a, b] for b in range(4)] for a in range(4)]
        low = [sum(gam[i][k] * v[k] for k in range(3)) for i in range(3)]
        S = [torch.zeros_like(r)]
        for i in range(3):
            s = -T[0][0] * al * da[i]
            for j in range(3):
                s = s + r * h * W * W * low[j] / al * db[i][j]
                for k in range(3):
                    s = s + (T[0][0] * 0.5 * be[j] * be[k] + T[0][j + 1] * be[k] + 0.5 * T[j + 1][k + 1]) * dg[i][j][k]
            S.append(s)
        e = torch.zeros_like(r)
        for i in range(3):
            e = e - T[0][0] * be[i] * da[i] - T[0][i + 1] * da[i]
            for j in range(3):
                e = e + (T[0][0] * be[i] * be[j] + 2.0 * T[0][i + 1] * be[j] + T[i + 1][j + 1]) * K[i][j]
        return al * sg * torch.stack(S + [e])


def _limited(ul, um, ur, limiter):
    dl, dr = um - ul, ur - um
    tiny = torch.full_like(dl, 1e-5)
    r = torch.where(dl.abs() < 1e-5, tiny, dl) / torch.where(dr.abs() < 1e-5, tiny, dr)
    a = r.clamp(min=0.0)
    xi = 2.0 / (1.0 + a)
    if limiter == SUPERBEE:
        phi = torch.where(a < 0.5, 2.0 * a, torch.where(a < 1.0, torch.ones_like(a),
                                                        torch.minimum(torch.minimum(a, xi), torch.full_like(a, 2.0))))
    elif limiter == VANLEER:
        phi = torch.minimum(2.0 * a / (1.0 + a), xi)
    else:
        phi = torch.where(a < 1.0, a, xi)
    return 0.5 * (dl + dr) * torch.where(r < 0.0, torch.zeros_like(phi), phi)


def _ghosts(q, k, periodic):
    """k ghost cells on each side of the last dimension: mirrored or wrapped."""
    if periodic:
        return torch.cat([q[..., -k:], q, q[..., :k]], -1)
    return torch.cat([q[..., :k].flip(-1), q, q[..., -k:].flip(-1)], -1)


def _sweep(sys, p, axis, dt, dx, order, limiter, periodic, on=None):
    q = p if axis == 0 else p.transpose(-1, -2)
    n = q.shape[-1]
    e = _ghosts(q, 2, periodic)
    along = dx * torch.arange(-2, n + 2, device=p.device, dtype=torch.float64)
    line = dx * torch.arange(q.shape[-2], device=p.device, dtype=torch.float64)[:, None]

    def at(lo, hi, shift=0.0):
        c = along[lo:len(along) + hi] + shift
        return (c, line) if axis == 0 else (line, c)

    U = sys.cons(e, at(0, 0))
    if order == 2:
        um, half = U[..., 1:-1], 0.5 * dx
        s = _limited(U[..., :-2], um, U[..., 2:], limiter)
        lo, hi = um - 0.5 * s, um + 0.5 * s
        ev = 0.5 * dt / dx * (sys.flux(lo, axis, at(1, -1, -half)) - sys.flux(hi, axis, at(1, -1, half)))
        left, right = sys.prim(hi + ev, at(1, -1, half))[..., :-1], sys.prim(lo + ev, at(1, -1, -half))[..., 1:]
    else:
        left, right = e[..., 1:-2], e[..., 2:-1]
    uL, uR = sys.cons(left, at(1, -2)), sys.cons(right, at(2, -1))
    fL, fR = sys.flux(uL, axis, at(1, -2)), sys.flux(uR, axis, at(2, -1))
    mid = 0.5 * (uL + uR + dt / dx * (fL - fR))
    F = 0.5 * (0.5 * (fL + fR + dx / dt * (uL - uR)) + sys.flux(mid, axis, at(2, -1, -0.5 * dx)))
    new = sys.prim(U[..., 2:-2] + dt / dx * (F[..., :-1] - F[..., 1:]), at(2, -2))
    new = new if axis == 0 else new.transpose(-1, -2)
    return new if on is None else torch.where(on, new, p)


def _rule(dt, t, t_final, it):
    dt = dt * 0.2 if it <= 5 else dt
    return t_final - t if t + dt > t_final else dt


def _step(sys, p, dt, dx, order, limiter, periodic, on=None):
    if p.shape[1] == 1:
        return _sweep(sys, p, 0, dt, dx, order, limiter, periodic, on)
    p = _sweep(sys, p, 0, 0.5 * dt, dx, order, limiter, periodic, on)
    p = _sweep(sys, p, 1, dt, dx, order, limiter, periodic, on)
    return _sweep(sys, p, 0, 0.5 * dt, dx, order, limiter, periodic, on)


def _solve(sys, p, case, dx):
    dims, t, it = (1 if p.shape[1] == 1 else 2), 0.0, 0
    t_final = case.get("t_final", FOREVER)
    while t < t_final and it != case["steps"]:
        dt = _rule(CFL * dx / float(sys.speed(p, dims).max()), t, t_final, it)
        p = _step(sys, p, dt, dx, case["order"], case["limiter"], case["periodic"])
        t, it = t + dt, it + 1
    return p


def _near(flag, reach):
    """Whether a cell or one within `reach` along either axis is flagged (flag has that border)."""
    ny, nx = flag.shape[0] - 2 * reach, flag.shape[1] - 2 * reach
    out = flag[reach:reach + ny, reach:reach + nx].clone()
    for d in range(-reach, reach + 1):
        out |= flag[reach + d:reach + d + ny, reach:reach + nx] | flag[reach:reach + ny, reach + d:reach + d + nx]
    return out


def _source_step(sys, p, dt, dx, parts, on):
    """Classical Runge-Kutta on the source with the reference's fractional sweeps between the stages."""
    ny, nx = p.shape[1:]
    x = dx * torch.arange(nx, device=p.device, dtype=torch.float64)
    y = dx * torch.arange(ny, device=p.device, dtype=torch.float64)[:, None]
    e = _ghosts(_ghosts(p, 1, False).transpose(-1, -2), 1, False).transpose(-1, -2)
    here, sides = (x, y), {}
    for axis in (0, 1):
        for s in (-1, 1):
            q = e[:, 1:-1, 1 + s:1 + s + nx] if axis == 0 else e[:, 1 + s:1 + s + ny, 1:-1]
            pos = (x + s * dx, y) if axis == 0 else (x, y + s * dx)
            sides[axis, s] = (sys.cons(sys.prim(sys.cons(q, pos), pos), pos), pos)

    def fraction(q, f, axis):
        (ul, pl), (ur, pr) = sides[axis, -1], sides[axis, 1]
        um = sys.cons(q, here)
        s = _limited(ul, um, ur, VANLEER)
        return sys.prim(um + f * dt / dx * (sys.flux(um - 0.5 * s, axis, pl) - sys.flux(um + 0.5 * s, axis, pr)), here)

    u = sys.cons(p, here)
    k = [dt * sys.source(u, here, parts)]
    for stage in range(3):
        fx, fy = (0.25, 0.5) if stage < 2 else (0.5, 1.0)
        q = sys.prim(u + (0.5 if stage < 2 else 1.0) * k[-1], here)
        q = fraction(fraction(fraction(q, fx, 0), fy, 1), fx, 0)
        k.append(dt * sys.source(sys.cons(q, here), here, parts))
    new = sys.prim(u + (k[0] + 2.0 * k[1] + 2.0 * k[2] + k[3]) / 6.0, here)
    return torch.where(on, new, p)


def _solve_gr(sys, p, case, dx):
    ny, nx = p.shape[1:]
    x = dx * torch.arange(-2, nx + 2, device=p.device, dtype=torch.float64)
    y = dx * torch.arange(-2, ny + 2, device=p.device, dtype=torch.float64)[:, None]
    out = sys.excised(x, y)
    sweep_on, source_on = ~_near(out, 2), ~_near(out[1:-1, 1:-1], 1)
    parts = sys.source_parts(x[2:-2], y[2:-2])
    t = 0.0
    for it in range(case["steps"]):
        dt = _rule(CFL * dx / float(sys.grid_speed(p).max()), t, FOREVER, it)
        p = _source_step(sys, p, 0.5 * dt, dx, parts, source_on)
        p = _step(sys, p, dt, dx, 2, case["limiter"], False, sweep_on)
        p = _source_step(sys, p, 0.5 * dt, dx, parts, source_on)
        t += dt
    return p


def _steep(u, dx, limit):
    """Cells with a conserved one-sided difference of at least `limit` (u has one border cell)."""
    c = u[:, 1:-1, 1:-1]
    near = (u[:, :-2, 1:-1], u[:, 2:, 1:-1], u[:, 1:-1, :-2], u[:, 1:-1, 2:])
    return torch.stack([((c - v) / dx).abs().amax(0) >= limit for v in near]).any(0)


def _border(u):
    return _ghosts(_ghosts(u, 1, False).transpose(-1, -2), 1, False).transpose(-1, -2)


def _twice(f):
    return f.repeat_interleave(2, -1).repeat_interleave(2, -2)


def _amr(sys, p, case, dx):
    t, fit, t_final, order = 0.0, 0, case["t_final"], case["order"]
    fine = _twice(p)
    con = torch.ones_like(p[0], dtype=torch.bool)
    fon = torch.zeros_like(fine[0], dtype=torch.bool)

    def restricted():
        u = sys.cons(fine, None)
        return sys.prim(0.25 * (u[:, ::2, ::2] + u[:, ::2, 1::2] + u[:, 1::2, ::2] + u[:, 1::2, 1::2]), None)

    while t < t_final:
        hit = _steep(_border(sys.cons(p, None)), dx, case["tol"])
        con, fon = con & ~hit, fon | _twice(hit)
        dt = _rule(CFL * dx / float(sys.speed(p, 2).max()), t, t_final, fit)
        p = _step(sys, p, dt, dx, order, VANLEER, False, con)
        if bool(fon.any()):
            ft = t
            while ft < t + dt - 1e-4:
                fdt = _rule(CFL * (0.5 * dx) / float(sys.speed(fine, 2).max()), ft, t + dt, fit)
                fine = _step(sys, fine, fdt, 0.5 * dx, order, VANLEER, False, fon)
                ft, fit = ft + fdt, fit + 1
        else:
            fit += 1
        t += dt
        p = torch.where(con, p, restricted())
        fine = torch.where(fon, fine, _twice(p))
        steep = _steep(_border(sys.cons(fine, None)), dx, 0.5 * case["tol"])[1::2, 1::2]
        calm = ~steep & fon[::2, ::2]
        fon, con = fon & ~_twice(calm), con | calm
        p = torch.where(calm, restricted(), p)
    return p, fine, con, fon


def _gradient(sys, p, case, dx, target):
    p0 = p.clone().requires_grad_(True)
    q, t, dts = p0, 0.0, []
    args = (dx, case["order"], case["limiter"], case["periodic"])
    for it in range(case["steps"]):
        with torch.no_grad():
            dt = _rule(CFL * dx / float(sys.speed(q, 2).max()), t, FOREVER, it)
        for axis, f in ((0, 0.5), (1, 1.0), (0, 0.5)):
            q = checkpoint(_sweep, sys, q, axis, f * dt, *args, use_reentrant=False)
        t += dt
        dts.append(dt)
    loss = 0.5 * ((q[0] - target) ** 2).sum()
    grad, = torch.autograd.grad(loss, p0)
    return float(loss.detach()), grad, torch.tensor(dts, dtype=torch.float64)


def exact(case, seed):
    if case["kind"] == "batch":
        sys = Newton(case)
        out = []
        for c, sh in zip(_batch_cells(case, seed), _batch_shapes(case, seed)):
            q = _solve(sys, c.permute(2, 0, 1).contiguous(), case, 1.0 / sh[-1])
            out.append(q.permute(1, 2, 0).reshape(sh + (5,)))
        return out
    sys = {"newton": Newton, "sr": Special, "gr": BlackHole}[case["system"]](case)
    cells, dx = _cells(case, seed), _dx(case)
    p = cells.permute(2, 0, 1).contiguous()
    if case["kind"] == "adjoint":
        loss, grad, dts = _gradient(sys, p, case, dx, _target(case, seed))
        return {"loss": loss, "grad": grad.permute(1, 2, 0).contiguous(), "dts": dts}
    with torch.no_grad():
        if case["kind"] == "amr":
            p, fine, con, fon = _amr(sys, p, case, dx)
            return {"coarse": p.permute(1, 2, 0).contiguous(), "fine": fine.permute(1, 2, 0).contiguous(),
                    "coarse_on": con, "fine_on": fon}
        p = (_solve_gr if sys.coords else _solve)(sys, p, case, dx)
    out = p.permute(1, 2, 0).contiguous()
    return out[0] if case["kind"] == "static" and case["ny"] == 0 else out
