"""What the framework is timed on: the work of a quasi-static simulation and
of an inversion for its coefficients, through the calls that such a program
makes.

A case is a dict of plain values.  ``kind`` is one of

* ``solve``    one projection solve on a handle that is kept: right-hand side
               and start guess in, V-cycles to a tolerance, solution out
               (``op``: shared stencil, Lame fields, or per-node stencils);
* ``step``     the drivers' projection step: divergence of the stresses,
               v_cycle() / l2_error_all() to the drivers' tolerance and two
               more cycles, stress update;
* ``frame``    a moving frame: a new shared stencil (full 3x3 blocks), the
               hierarchy rebuilt, a warm-started solve;
* ``invert``   one step of an inversion for the coefficients: a solve with new
               Lame fields and its gradients, through the autograd function;
* ``advect``   the advection step before the projection;
* ``output``   the values of the fields that a frame of output files holds.

Inputs are made on the GPU from the seed: stresses N(0, 1e-3), lognormal
coefficients (sigma 0.3), deviatoric stresses from half to 1.15 of the yield
stress, as the benchmark and the tests have them.
"""
import math

import torch

import stzpp_gb300 as sg
from stzpp_gb300 import advect
from stzpp_gb300.autograd import ProjectionSolver

PLATES = (True, True, False)     # periodic x and y, Dirichlet plates in z
BOX = (False, False, False)      # Dirichlet on every face


def listed():
    return [
        # the benchmark: the largest solve of the drivers, mixed precision, V(2,4) on every level
        dict(name="solve_mixed_256", kind="solve", op="const", m=256, n=256, o=257, precision="mixed", v_down=2,
             v_up=4, growth=False, bottom="direct", tol=1e-10),
        # the smallest: the 33^3 problem, where launches and synchronisations count
        dict(name="solve_mixed_32", kind="solve", op="const", m=32, n=32, o=33, precision="mixed", v_down=2, v_up=2,
             growth=True, bottom="direct", tol=1e-10),
        # plain FP64 with the reference's cycle (growing sweeps), a ragged middle size
        dict(name="solve_fp64_160x96x129", kind="solve", op="const", m=160, n=96, o=129, precision="fp64", v_down=2,
             v_up=2, growth=True, bottom="direct", tol=1e-10),
        # variable coefficients on a kept operator, as in a sequence of solves with fixed fields
        dict(name="solve_lame_mixed_128", kind="solve", op="lame", m=128, n=128, o=129, precision="mixed", v_down=2,
             v_up=2, growth=False, bottom="direct", tol=1e-10),
        dict(name="solve_lame_fp64_64x96x50", kind="solve", op="lame", m=64, n=96, o=50, precision="fp64", v_down=2,
             v_up=2, growth=True, bottom="direct", tol=1e-10),
        # a caller's own assembled stencils on a closed box, odd sizes, the reference's Gauss-Seidel bottom
        dict(name="solve_points_fp64_49x41x33", kind="solve", op="points", m=49, n=41, o=33, precision="fp64",
             v_down=2, v_up=2, growth=True, bottom="gs", tol=1e-10),
        # one projection step as the drivers call it
        dict(name="step_mixed_192", kind="step", m=192, n=192, o=193, precision="mixed", v_down=2, v_up=2,
             growth=True),
        # a new stencil each step, as in a deforming frame
        dict(name="frame_mixed_128", kind="frame", m=128, n=128, o=129, precision="mixed", v_down=2, v_up=4,
             growth=False, tol=1e-10),
        # forward and backward with new coefficients, as each step of an inversion has them
        dict(name="invert_mixed_64", kind="invert", m=64, n=64, o=65, precision="mixed", tol=1e-10),
        # the advection step at the benchmark's size, and a small ragged one
        dict(name="advect_256", kind="advect", m=256, n=256, o=256, dt=200.0, top=1.15),
        dict(name="advect_48x40x24", kind="advect", m=48, n=40, o=24, dt=200.0, top=1.15),
        # the fields of one output frame
        dict(name="output_192", kind="output", m=192, n=192, o=192),
    ]


def _bottom(m, n, o):
    """Nodes of the coarsest level: halved while there are over 1024 and the periodic sides stay even."""
    while m * n * o > 1024 and m % 4 == 0 and n % 4 == 0:
        m, n, o = m // 2, n // 2, (o + 2) // 2
    return m * n * o


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(hi, bottom=2048):
        """Extents up to hi with sides within a factor of two; the periodic ones
        (x, y) are such that the hierarchy can halve them down to a small bottom."""
        even = [v for v in (16, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256) if v <= hi]
        while True:
            m, n = rng.choice(even), rng.choice(even)
            o = size(max(17, m // 2), min(hi, 2 * m) + 1)
            if max(m, n) <= 2 * min(m, n) and _bottom(m, n, o) <= bottom:
                return dict(m=m, n=n, o=o)

    def cycle():
        v_down, v_up = rng.choice([(2, 2), (2, 4), (2, 3), (1, 2)])
        return dict(v_down=v_down, v_up=v_up, growth=rng.random() < 0.5)

    kind = rng.choice(["const", "const", "const", "lame", "lame", "points", "step", "step", "frame", "frame", "invert",
                       "invert", "advect", "advect", "output"])
    if kind == "const":
        mixed = rng.random() < 0.6
        hi = 256 if mixed else 128
        return dict(kind="solve", op="const", precision="mixed" if mixed else "fp64", bottom="direct",
                    tol=rng.choice([1e-8, 1e-10]), **grid(hi), **cycle())
    if kind == "lame":
        mixed = rng.random() < 0.6
        hi = 128 if mixed else 96
        return dict(kind="solve", op="lame", precision="mixed" if mixed else "fp64", bottom="direct",
                    tol=rng.choice([1e-8, 1e-10]), **grid(hi, 600), **cycle())
    if kind == "points":
        return dict(kind="solve", op="points", m=size(17, 65), n=size(17, 65), o=size(17, 65),
                    precision=rng.choice(["mixed", "fp64"]), bottom=rng.choice(["gs", "direct"]), tol=1e-10,
                    v_down=2, v_up=2, growth=True)
    if kind == "step":
        mixed = rng.random() < 0.7
        return dict(kind="step", precision="mixed" if mixed else "fp64", **grid(192 if mixed else 128), **cycle())
    if kind == "frame":
        return dict(kind="frame", precision="mixed", tol=1e-10, **grid(128), **cycle())
    if kind == "invert":
        return dict(kind="invert", precision=rng.choice(["mixed", "mixed", "fp64"]), tol=1e-10, **grid(64, 600))
    if kind == "advect":
        return dict(kind="advect", m=size(16, 256), n=size(16, 256), o=size(16, 256), dt=200.0,
                    top=round(rng.uniform(0.9, 1.2), 3))
    return dict(kind="output", m=size(24, 256), n=size(24, 256), o=size(24, 256))


# ------------------------------------------------------------------ inputs
def _dims(c):
    return c["m"], c["n"], c["o"]


def _periodic(c):
    return BOX if c.get("op") == "points" else PLATES


def _spacing(c):
    """The same spacing on every axis, 1/m, so that a case of any shape has cubes for cells."""
    return (1.0 / c["m"],) * 3


def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + k)


def _normal(shape, std, gen):
    return torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda") * std


def _cells(c):
    """Cells per axis, z first."""
    return tuple(d if p else d - 1 for d, p in zip(_dims(c), _periodic(c)))[::-1]


def _stress(c, seed):
    """Cell tensors (cells_z, cells_y, cells_x, 6), components s11 s12 s13 s22 s23 s33."""
    return _normal(_cells(c) + (6,), 1e-3, _gen(seed))


def _divergence(s, dims, per, h):
    """Node divergence (o, n, m, 3) of a cell tensor field: differences of the
    8 cells about a node; 0 on the Dirichlet faces."""
    full = torch.zeros(dims[2], dims[1], dims[0], 6, dtype=s.dtype, device=s.device)
    full[:s.shape[0], :s.shape[1], :s.shape[2]] = s

    def diff(a, axis):   # axis 0, 1, 2: x, y, z
        for d in range(3):
            b = torch.roll(a, 1, 2 - d)
            a = (a - b) / h[d] if d == axis else 0.5 * (a + b)
        return a

    r = torch.empty(full.shape[:3] + (3,), dtype=s.dtype, device=s.device)
    row = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
    for k in range(3):
        r[..., k] = diff(full[..., row[k][0]], 0) + diff(full[..., row[k][1]], 1) + diff(full[..., row[k][2]], 2)
    r[~_interior(dims, per)] = 0.0
    return r


def _interior(dims, per):
    inside = torch.ones(dims[2], dims[1], dims[0], dtype=torch.bool, device="cuda")
    for axis in range(3):
        if not per[axis]:
            inside.select(2 - axis, 0).fill_(False)
            inside.select(2 - axis, dims[axis] - 1).fill_(False)
    return inside


def _rhs(c, seed):
    return _divergence(_stress(c, seed), _dims(c), _periodic(c), _spacing(c)).reshape(-1, 3).contiguous()


def _log_mu(c, seed):
    """log mu per node, N(0, 0.3)."""
    return _normal((c["o"], c["n"], c["m"]), 0.3, _gen(seed, 1)).reshape(-1)


def _shear(seed, k):
    """The frame's transform at step k: the identity with a few per cent of shear and stretch."""
    gen = torch.Generator().manual_seed(1000003 * seed + 7)
    return torch.eye(3, dtype=torch.float64) + (0.05 + 0.01 * k) * torch.randn(3, 3, generator=gen, dtype=torch.float64)


def _frame_stencil(T, lam, mu, h):
    """27 x 9 stencil and fix block of -(mu lap + (lam + mu) grad div) in a
    frame where d/dx_i = sum_a T[i][a] d/dq_a: second differences on the faces,
    four-point ones on the edges, full blocks."""
    base = torch.zeros(3, 3, 3, 3, 3, dtype=torch.float64)   # dz, dy, dx, row, column
    for a in range(3):
        for b in range(3):
            block = mu * torch.eye(3, dtype=torch.float64) * float(T[:, a] @ T[:, b])
            block = block + 0.5 * (lam + mu) * (torch.outer(T[:, a], T[:, b]) + torch.outer(T[:, b], T[:, a]))
            for sa in (-1, 1):
                if a == b:
                    d = [1, 1, 1]
                    d[a] += sa
                    base[d[2], d[1], d[0]] += block / h[a] ** 2
                    base[1, 1, 1] -= block / h[a] ** 2
                    continue
                for sb in (-1, 1):
                    d = [1, 1, 1]
                    d[a] += sa
                    d[b] += sb
                    base[d[2], d[1], d[0]] += sa * sb * block / (4 * h[a] * h[b])
    fix = torch.eye(3, dtype=torch.float64) * float(base[1, 1, 1].diagonal().min())
    return (-base).reshape(27, 9).numpy(), fix.reshape(9).numpy()


def _stencil(c, seed):
    if c["kind"] == "frame":
        return _frame_stencil(_shear(seed, 1), 2.0, 1.0, _spacing(c))
    return sg.elastic_stencil(1.0, 2.0, *_spacing(c))


def _lame_entries(mu, lam, h):
    """The variable-coefficient operator -div(mu (grad u + grad u^T) + lam
    (div u) I) as (offset, row, column, coefficient field): coefficients at
    the faces' midpoints, node values on the edges."""
    def at(f, d):
        return torch.roll(f, (-d[2], -d[1], -d[0]), (0, 1, 2))

    entries, centre = [], [0.0, 0.0, 0.0]
    for axis in range(3):
        for s in (-1, 1):
            d = [0, 0, 0]
            d[axis] = s
            mu_f, lam_f = 0.5 * (mu + at(mu, d)), 0.5 * (lam + at(lam, d))
            for k in range(3):
                v = (lam_f + 2 * mu_f if k == axis else mu_f) / h[axis] ** 2
                entries.append((tuple(d), k, k, -v))
                centre[k] = centre[k] + v
    entries += [((0, 0, 0), k, k, centre[k]) for k in range(3)]
    for r in range(3):
        for k in range(3):
            for sr in (-1, 1):
                for sk in (-1, 1):
                    if r == k:
                        continue
                    d, dr, dk = [0, 0, 0], [0, 0, 0], [0, 0, 0]
                    d[r], d[k], dr[r], dk[k] = sr, sk, sr, sk
                    entries.append((tuple(d), r, k, -sr * sk * (at(lam, dr) + at(mu, dk)) / (4 * h[r] * h[k])))
    fix = -2 * ((lam + 2 * mu) / h[0] ** 2 + mu / h[1] ** 2 + mu / h[2] ** 2)
    return entries, fix


def _points(mu, lam, dims, per, h):
    """The same operator as per-node stencils (npts, 27, 9)."""
    shape = dims[::-1]
    entries, fix = _lame_entries(mu.reshape(shape), lam.reshape(shape), h)
    inside = _interior(dims, per)
    A = torch.zeros(shape + (27, 9), dtype=torch.float64, device=mu.device)
    for d, r, k, v in entries:
        A[..., 13 + d[0] + 3 * d[1] + 9 * d[2], 3 * r + k] = torch.where(inside, v, torch.zeros_like(v))
    for k in range(3):
        A[..., 13, 4 * k] = torch.where(inside, A[..., 13, 4 * k], fix)
    return A.reshape(-1, 243).contiguous()


def _handle(c):
    return sg.Multigrid(_dims(c), _periodic(c), precision=c["precision"], v_down=c["v_down"], v_up=c["v_up"],
                        sweep_growth=c["growth"], bottom=c.get("bottom", "direct"),
                        stream=torch.cuda.current_stream().cuda_stream)


# the simulation's parameters, in units of the yield stress and the shear-wave time
LAM, MU, DT = 2.0, 1.0, 1.0
STZ = dict(mu=44.01, sy=1.0, tau0=2.472e-8, c0=0.4, eps0=0.3, delta=0.381, omega=1.345, bath_temp=0.01905,
           chi_inf=0.04286, ez=1.0)
OUTPUT_MODES = (0, 1, 2, 9, 10, 12)   # velocities, pressure, deviatoric stress, effective temperature


def _grid_fields(c, seed):
    """Members of the ghosted grid: velocities N(0, 1e-3), stresses of random
    direction with deviatoric magnitudes from 0.5 to `top` of the yield
    stress, effective temperatures about 550 K; ghosts periodic in x and y,
    random in z."""
    g, gen = advect.NGHOST, _gen(seed)
    dims = _dims(c)
    shape = tuple(v + 2 * g for v in dims[::-1])
    f = {}
    for k in advect.INPUTS:
        f[k] = _normal(shape, 1e-3 if k in "uvw" else 15 / 21000 if k == "chi" else 1.0, gen)
    f["chi"] += 550 / 21000
    p = -(f["s11"] + f["s22"] + f["s33"]) / 3
    dev = torch.sqrt(0.5 * ((f["s11"] + p) ** 2 + (f["s22"] + p) ** 2 + (f["s33"] + p) ** 2) + f["s12"] ** 2
                     + f["s13"] ** 2 + f["s23"] ** 2)
    target = 0.5 + (c.get("top", 1.15) - 0.5) * torch.rand(shape, generator=gen, dtype=torch.float64, device="cuda")
    for k in ("s11", "s12", "s13", "s22", "s23", "s33"):
        f[k] = f[k] * target / dev
    f["ad_dpl"] = 1e-3 * torch.rand(shape, generator=gen, dtype=torch.float64, device="cuda")
    for t in f.values():
        for axis, n in ((2, dims[0]), (1, dims[1])):
            t.narrow(axis, 0, g).copy_(t.narrow(axis, n, g).clone())
            t.narrow(axis, n + g, g).copy_(t.narrow(axis, g, g).clone())
    return {k: t.reshape(-1).contiguous() for k, t in f.items()}


def _stz(c):
    return dict(STZ, diff_l=1.5 / c["m"])


# ------------------------------------------------------------------ the path
def prepare(case, seed):
    c = case
    if c["kind"] == "advect":
        f = _grid_fields(c, seed)
        for k in advect.OUTPUTS:
            f.setdefault(k, torch.zeros_like(f["u"]))
        work = torch.empty(advect.work_size(*_dims(c)), dtype=torch.float64, device="cuda")
        return dict(case=c, fields=f, work=work)
    if c["kind"] == "output":
        return dict(case=c, fields=_grid_fields(c, seed))
    if c["kind"] == "invert":
        solver = ProjectionSolver(_dims(c), PLATES, _spacing(c), precision=c["precision"], tol=c["tol"])
        target = _normal((c["m"] * c["n"] * c["o"], 3), 1e-3, _gen(seed, 2))
        return dict(case=c, solver=solver, b=_rhs(c, seed), log_mu=_log_mu(c, seed), target=target)
    mg = _handle(c)
    state = dict(case=c, mg=mg)
    state["zero"] = torch.zeros(mg.npts, 3, dtype=torch.float64, device="cuda")
    if c["kind"] == "step":
        state["stress"] = _stress(c, seed)
        state["new_stress"] = torch.empty_like(state["stress"])
        stencil, fix = _stencil(c, seed)
        # the drivers' stopping rule: sum of |r|^4 against the centre coefficient
        state["stop"] = (2.220446049250313e-16 * abs(float(stencil.reshape(27, 9)[13, 0])) * 1e3) ** 2
        mg.setup_matrices(stencil, fix)
        return state
    state["b"], state["x"] = _rhs(c, seed), torch.empty_like(state["zero"])
    if c["kind"] == "frame":
        # the step before: another frame, solved
        mg.setup_matrices(*_frame_stencil(_shear(seed, 0), LAM, MU, _spacing(c)))
        mg.setup_fields(x=state["zero"], r=state["b"])
        mg.solve(1e-10, 200)
        state["before"] = mg.get_x(torch.empty_like(state["zero"]))
        state["stencil"], state["fix"] = _stencil(c, seed)
        return state
    if c["op"] == "const":
        mg.setup_matrices(*_stencil(c, seed))
        return state
    mu = torch.exp(_log_mu(c, seed))
    if c["op"] == "lame":
        mg.setup_matrices(mu=mu, lam=2 * mu, spacing=_spacing(c))
    else:
        mg.setup_matrices(points=_points(mu, 2 * mu, _dims(c), BOX, _spacing(c)))
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "advect":
        f = state["fields"]
        f["cchi"].zero_()   # the caller has merged the last step's changes
        advect.advection_step(f, _dims(c), _spacing(c), _stz(c), c["dt"], work=state["work"], wait=False)
        return {k: f[k] for k in advect.OUTPUTS}
    if c["kind"] == "output":
        return [advect.cube_values(state["fields"], _dims(c), mode) for mode in OUTPUT_MODES]
    if c["kind"] == "invert":
        b = state["b"].detach().requires_grad_(True)
        log_mu = state["log_mu"].detach().requires_grad_(True)
        mu = torch.exp(log_mu)
        u = state["solver"](b, mu, 2 * mu)
        loss = ((u - state["target"]) ** 2).sum()
        gb, gl = torch.autograd.grad(loss, (b, log_mu))
        return dict(u=u.detach(), loss=loss.detach(), grad_b=gb, grad_log_mu=gl)
    mg = state["mg"]
    if c["kind"] == "step":
        stress = state["new_stress"].copy_(state["stress"])
        mg.set_rhs_divergence(stress, _spacing(c))
        mg.set_x(state["zero"])
        for _ in range(200):
            mg.v_cycle()
            if mg.l2_error_all() <= state["stop"]:
                break
        mg.v_cycle()
        mg.v_cycle()
        return dict(stress=stress, proj_mag=mg.stress_update(stress, LAM, MU, DT, _spacing(c)))
    if c["kind"] == "frame":
        mg.setup_matrices(state["stencil"], state["fix"])
        mg.setup_fields(x=state["before"], r=state["b"])
    else:
        mg.setup_fields(x=state["zero"], r=state["b"])
    mg.solve(c["tol"], 200)
    return mg.get_x(state["x"])


def work(case):
    """Bytes: the arrays that go in and come out, once.  Flops: for a solve ten
    cycles of six passes over the nodes of all levels (8/7 of the finest), a
    pass being the products of the operator's non-zero entries."""
    c = case
    nodes = c["m"] * c["n"] * c["o"]
    if c["kind"] == "advect":
        return dict(bytes=21 * 8 * nodes, flops=500 * nodes)
    if c["kind"] == "output":
        return dict(bytes=(12 * 8 + 4 * len(OUTPUT_MODES)) * nodes, flops=40 * nodes)
    entries = 243 if c.get("op") == "points" else 171 if c["kind"] == "frame" else 45
    solve = 10 * 6 * nodes * 8 / 7 * 2 * entries
    if c["kind"] == "step":
        return dict(bytes=2 * 48 * nodes, flops=solve)
    if c["kind"] == "invert":
        return dict(bytes=(3 * 24 + 24 + 24 + 16) * nodes, flops=2 * solve)
    coef = dict(points=243 * 8, lame=16).get(c.get("op"), 0)
    return dict(bytes=(3 * 24 + coef) * nodes, flops=solve)


# ------------------------------------------------------------------ in 64 bits
class _Periodic:
    """Direct solver of a shared stencil, periodic in x and y, Dirichlet plates
    in z (zero there): a Fourier transform in x and y, block elimination in z."""

    def __init__(self, stencil, dims):
        self.m, self.n, self.o = dims
        A = torch.as_tensor(stencil, dtype=torch.float64).reshape(3, 3, 3, 3, 3).to("cuda", torch.complex128)
        kx = 2j * math.pi * torch.arange(self.m // 2 + 1, dtype=torch.float64, device="cuda") / self.m
        ky = 2j * math.pi * torch.arange(self.n, dtype=torch.float64, device="cuda") / self.n
        wx = [torch.exp(kx * (d - 1))[None, :, None, None] for d in range(3)]
        wy = [torch.exp(ky * (d - 1))[:, None, None, None] for d in range(3)]
        sym = [sum(A[dz, dy, dx] * wx[dx] * wy[dy] for dy in range(3) for dx in range(3)).reshape(-1, 3, 3)
               for dz in range(3)]
        self.low, diag, self.up = sym
        self.inv = []
        last = None
        for _ in range(self.o - 2):
            last = _inverse3(diag if last is None else diag - self.low @ (last @ self.up))
            self.inv.append(last)

    def solve(self, b):
        f = torch.fft.rfft2(b, dim=(1, 2)).reshape(self.o, -1, 3, 1)
        y = torch.zeros_like(f)
        for k in range(1, self.o - 1):
            y[k] = self.inv[k - 1] @ (f[k] - (self.low @ y[k - 1]))
        for k in range(self.o - 3, 0, -1):
            y[k] -= self.inv[k - 1] @ (self.up @ y[k + 1])
        return torch.fft.irfft2(y.reshape(self.o, self.n, -1, 3), s=(self.n, self.m), dim=(1, 2))


def _inverse3(a):
    r = [a[:, k] for k in range(3)]
    cols = torch.stack([torch.linalg.cross(r[(k + 1) % 3], r[(k + 2) % 3]) for k in range(3)], -1)
    return cols / (r[0] * cols[:, :, 0]).sum(-1)[:, None, None]


def _apply(entries, fix, inside, u):
    """A u with u of shape (o, n, m, 3)."""
    out = [0.0, 0.0, 0.0]
    for d, r, k, v in entries:
        out[r] = out[r] + v * torch.roll(u[..., k], (-d[2], -d[1], -d[0]), (0, 1, 2))
    return torch.where(inside[..., None], torch.stack(out, -1), fix[..., None] * u)


def _lame_solve(c, mu, lam, b):
    """u with A u = b for a b that is zero on the Dirichlet faces: conjugate
    gradients on the inner nodes, with the constant operator as the
    preconditioner where that has a direct solver."""
    shape, h = _dims(c)[::-1], _spacing(c)
    inside = _interior(_dims(c), _periodic(c))
    entries, fix = _lame_entries(mu.reshape(shape), lam.reshape(shape), h)
    if c.get("op") == "points":
        diag = torch.stack([v for d, r, k, v in entries if d == (0, 0, 0)], -1)

        def pre(r):
            return torch.where(inside[..., None], r / diag, 0.0)
    else:
        pre = _Periodic(_plain_stencil(float(mu.mean()), float(lam.mean()), h), _dims(c)).solve

    def A(v):
        return torch.where(inside[..., None], _apply(entries, fix, inside, v), 0.0)

    b = torch.where(inside[..., None], b.reshape(shape + (3,)), 0.0)
    x = torch.zeros_like(b)
    for _ in range(2):   # started again once from the true residual
        r = b - A(x)
        z = pre(r)
        p, rz = z.clone(), (r * z).sum()
        for it in range(2000):
            q = A(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if it % 8 == 7 and float(r.norm()) <= 1e-14 * float(b.norm()):
                break
            z = pre(r)
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
    return x, entries, fix, inside


def _plain_stencil(mu, lam, h):
    """The constant-coefficient stencil, from the frame's with the identity."""
    return _frame_stencil(torch.eye(3, dtype=torch.float64), lam, mu, h)[0]


def _exact_stress(c, stress, u):
    """stress + dt (lam tr(grad u) I + mu (grad u + grad u^T)) per cell, and
    the sum over the cells of half the squared norm of the increment."""
    h = _spacing(c)
    cells = stress.shape[:3]

    def d(k, axis):
        a = u[..., k]
        for e in range(3):
            up = torch.roll(a, -1, 2 - e)
            a = (up - a) / h[e] if e == axis else 0.5 * (up + a)
        return a[:cells[0], :cells[1], :cells[2]]

    g = [[d(k, a) for a in range(3)] for k in range(3)]
    tr = g[0][0] + g[1][1] + g[2][2]
    ds = [DT * ((LAM * tr if r == k else 0.0) + MU * (g[r][k] + g[k][r])) for r, k in
          ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
    mag = 0.5 * sum((1 if e in (0, 3, 5) else 2) * (s * s).sum() for e, s in enumerate(ds))
    return stress + torch.stack(ds, -1), mag


def _dev(s11, s12, s13, s22, s23, s33):
    p = -(s11 + s22 + s33) / 3
    return torch.sqrt(0.5 * ((s11 + p) ** 2 + (s22 + p) ** 2 + (s33 + p) ** 2) + s12 ** 2 + s13 ** 2 + s23 ** 2)


def _exact_output(c, seed):
    f, g, (m, n, o) = _grid_fields(c, seed), advect.NGHOST, _dims(c)
    f = {k: t.reshape(o + 2 * g, n + 2 * g, m + 2 * g) for k, t in f.items()}
    stress = [f[k] for k in ("s11", "s12", "s13", "s22", "s23", "s33")]
    values = [f["u"], f["v"], f["w"], -(f["s11"] + f["s22"] + f["s33"]) / 3, _dev(*stress), 21000 * f["chi"]]
    out = []
    for mode, v in zip(OUTPUT_MODES, values):
        inner = v[g:g + o + (mode <= 2), g:g + n, g:g + m]
        out.append(inner.permute(2, 1, 0).reshape(-1))   # x slowest, z fastest
    return out


def _exact_advect(c, seed):
    """The step's formulas on whole arrays: adaptive plastic sub-steps, ENO2
    advection, the Truesdell terms, the diffusion of chi."""
    g, (m, n, o), h, P, dt = advect.NGHOST, _dims(c), _spacing(c), _stz(c), c["dt"]
    shape = (o + 2 * g, n + 2 * g, m + 2 * g)
    f = {k: t.reshape(shape) for k, t in _grid_fields(c, seed).items()}

    def at(a, x=0, y=0, z=0):
        return a[g + z:g + z + o, g + y:g + y + n, g + x:g + x + m]

    def inner(v, before):
        out = before.clone()
        out[g:g + o, g:g + n, g:g + m] = v
        return out.reshape(-1)

    S = {k: at(f[k]) for k in ("s11", "s12", "s13", "s22", "s23", "s33")}
    sbar = _dev(*S.values())
    # plastic sub-steps of the cells above the yield stress
    at_yield = sbar > P["sy"]
    s0, c0 = sbar[at_yield], at(f["chi"])[at_yield]
    sa, ca, left = s0.clone(), c0.clone(), torch.full_like(s0, dt)
    live = torch.arange(s0.numel(), device=s0.device)
    while live.numel():
        s, x, t = sa[live], ca[live], left[live]
        e = P["omega"] * P["eps0"] * s
        rate = torch.exp(-P["ez"] / x) * 0.5 * (torch.exp((e - P["delta"]) / P["bath_temp"])
                                                + torch.exp(-(e + P["delta"]) / P["bath_temp"]))
        rate = torch.where(s >= P["sy"], rate * (1 - P["sy"] / s) / P["tau0"], 0.0)
        dp = 2 * P["mu"] * rate / P["sy"]
        F = 2 * rate * s * (P["chi_inf"] - x) / (P["sy"] * P["c0"])
        more = dp * t > 5e-4
        ts = torch.where(more, 5e-4 / dp.abs().clamp_min(1e-300), t)
        sa[live], ca[live], left[live] = s - ts * dp * P["sy"], x + ts * F, t - ts
        live = live[more]
    adapt, dchi = torch.zeros_like(sbar), torch.zeros_like(sbar)
    adapt[at_yield], dchi[at_yield] = 1 - sa / s0, ca - c0
    ad_new = adapt * 0.5 / P["mu"] * sbar

    def d(a, axis):   # of node values, at the cell
        for e in range(3):
            k = [0, 0, 0]
            k[e] = 1
            up = torch.roll(a, (-k[2], -k[1], -k[0]), (0, 1, 2))
            a = (up - a) / h[e] if e == axis else 0.5 * (up + a)
        return at(a)

    vel = [d(f[k], -1) for k in "uvw"]
    grad = [[d(f[k], a) for a in range(3)] for k in "uvw"]

    def advance(a):
        total = 0.0
        for axis in range(3):
            e = [0, 0, 0]

            def s(j):
                e[axis] = j
                return at(a, *e)
            f2p, fp, f0, fm, f2m = s(2), s(1), s(0), s(-1), s(-2)
            mid, fw, bk = (fp - 2 * f0 + fm).abs(), (f2p - 2 * fp + f0).abs(), (f0 - 2 * fm + f2m).abs()
            even = fp - fm
            neg = torch.where(mid > fw, -f2p + 4 * fp - 3 * f0, even)
            pos = torch.where(mid > bk, 3 * f0 - 4 * fm + f2m, even)
            total = total + vel[axis] * torch.where(vel[axis] < 0, neg, pos) * 0.5 * dt / h[axis]
        return total

    comp = (("s11", "s12", "s13"), ("s12", "s22", "s23"), ("s13", "s23", "s33"))
    tr = grad[0][0] + grad[1][1] + grad[2][2]
    zero = torch.zeros(shape, dtype=torch.float64, device="cuda")
    out = dict(sbar=inner(sbar, zero))
    trace = S["s11"] + S["s22"] + S["s33"]
    for r, k in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)):
        name = comp[r][k]
        trues = sum(S[comp[k][q]] * grad[r][q] + S[comp[r][q]] * grad[k][q] for q in range(3)) - S[name] * tr
        plast = -adapt * (S[name] - (trace / 3 if r == k else 0.0))
        out["c" + name] = inner(plast - advance(f[name]) + dt * trues, zero)
    # the sweep has the new ad_Dpl behind it and the old one ahead
    new = f["ad_dpl"].clone()
    new[g:g + o, g:g + n, g:g + m] = ad_new
    old = f["ad_dpl"]
    chi, diff = f["chi"], 0.0
    for axis in range(3):
        e, q = [0, 0, 0], [0, 0, 0]
        e[axis], q[axis] = 1, -1
        gD = 0.5 * (at(old, *e) - at(new, *q)) / h[axis]
        gc = 0.5 * (at(chi, *e) - at(chi, *q)) / h[axis]
        lc = (at(chi, *e) - 2 * at(chi) + at(chi, *q)) / h[axis] ** 2
        diff = diff + gD * gc + ad_new * lc
    out["cchi"] = inner(dchi - advance(chi) + P["diff_l"] ** 2 * diff / P["c0"], zero)
    out["ad_dpl"] = new.reshape(-1)
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "output":
        return _exact_output(c, seed)
    if c["kind"] == "advect":
        return _exact_advect(c, seed)
    dims = _dims(c)
    if c["kind"] == "step":
        stress = _stress(c, seed)
        b = _divergence(stress, dims, PLATES, _spacing(c))
        u = _Periodic(_plain_stencil(MU, LAM, _spacing(c)), dims).solve(b)
        new, mag = _exact_stress(c, stress, u)
        return dict(stress=new, proj_mag=float(mag))
    b = _rhs(c, seed).reshape(dims[::-1] + (3,))
    if c["kind"] == "frame":
        return _Periodic(_stencil(c, seed)[0], dims).solve(b).reshape(-1, 3)
    if c["kind"] == "solve" and c["op"] == "const":
        return _Periodic(_plain_stencil(MU, LAM, _spacing(c)), dims).solve(b).reshape(-1, 3)
    log_mu = _log_mu(c, seed)
    mu = torch.exp(log_mu)
    u, entries, fix, inside = _lame_solve(c, mu, 2 * mu, b)
    if c["kind"] == "solve":
        return u.reshape(-1, 3)
    # gradients of |u - target|^2: A^T w = 2 (u - target), -w . dA u
    target = _normal((mu.numel(), 3), 1e-3, _gen(seed, 2)).reshape(u.shape)
    gu = 2 * (u - target)
    w = _lame_solve(c, mu, 2 * mu, gu)[0]
    v = torch.zeros_like(u).requires_grad_(True)
    (on_faces,) = torch.autograd.grad((_apply(entries, fix, inside, v) * w).sum(), v)
    w = torch.where(inside[..., None], w, (gu - on_faces) / fix[..., None])
    log_mu.requires_grad_(True)
    field = torch.exp(log_mu).reshape(dims[::-1])
    entries, fix = _lame_entries(field, 2 * field, _spacing(c))
    (grad,) = torch.autograd.grad(-(_apply(entries, fix, inside, u) * w).sum(), log_mu)
    return dict(u=u.reshape(-1, 3), loss=((u - target) ** 2).sum(), grad_b=w.reshape(-1, 3), grad_log_mu=grad)
