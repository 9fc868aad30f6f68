"""The framework's workloads as timed cases: the fluid step in 2D and 3D, its
parts (conjugate gradient, advection), many grids at once, the learned
pressure network (forward and training) and the wavelet transforms, each
through the package's public entry points.

A step case advances one frame: the frame's fields are copied into the
working fields (frames come from elsewhere, and every pass then does the
same work), then one step runs.  Every sample of `draw` is of the same kinds.
"""

import itertools
import math

import numpy as np
import torch

import panopaea_gb300 as pg
from panopaea_gb300 import wavelet

KINDS = ("example_2d", "plume_2d", "step_3d", "batch_2d", "cg", "transport_3d", "network_3d", "train_3d", "wavelet_2d")


def listed():
    return [
        # The reference example's own step (examples/dec_fluid.rs): 128^2
        # doubles, inflow box, obstacle, at most 100 plain CG iterations.
        dict(name="example_2d_128_f64", kind="example_2d", h=128, w=128),
        # The 256^2 buoyant plume, multigrid CG in refinement to 1e-5.
        dict(name="plume_2d_256", kind="plume_2d", h=256, w=256, circles=0),
        # A small interactive room with box obstacles.
        dict(name="room_3d_64", kind="step_3d", d=64, h=64, w=64, shape="boxes"),
        # The same with odd sides: rows that start on no vector boundary.
        dict(name="room_3d_93x118x75", kind="step_3d", d=93, h=118, w=75, shape="boxes"),
        # The headline configuration: 256^3 filtered noise, projection to 1e-6.
        dict(name="noise_3d_256", kind="step_3d", d=256, h=256, w=256, shape="open"),
        # The largest single grid: 512^3 around a solid sphere, buoyant smoke.
        dict(name="sphere_3d_512", kind="step_3d", d=512, h=512, w=512, shape="sphere"),
        # Many independent 2D plumes with circles and boundary sources at once.
        dict(name="batch_2d_256", kind="batch_2d", count=256, lo=64, hi=512, unit=32),
        # The reference's plain CG, its 100 iterations, on a 3D grid.
        dict(name="cg_3d_160x144x176", kind="cg", d=160, h=144, w=176, precond="none", dtype="f32"),
        # Velocity and density transport alone, second order in the density.
        dict(name="transport_3d_192", kind="transport_3d", d=192, h=192, w=192, scheme=1, dtype="f32"),
        # The learned network on one 128^3 right-hand side: its output, which
        # the guess scales and the solve starts from.
        dict(name="network_3d_128", kind="network_3d", d=128, h=128, w=128),
        # One training sample of the network: forward, backward, gradients out.
        dict(name="train_3d_96", kind="train_3d", d=96, h=96, w=96),
        # Wavelet analysis and synthesis of a 2D field.
        dict(name="wavelet_2d_1024", kind="wavelet_2d", h=1024, w=1024, levels=5, filter=wavelet.BIOR22),
    ]


def draw(rng):
    def side(lo, hi, unit=1):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return max(lo, min(hi, int(round(v / unit)) * unit))

    kind = rng.choice(KINDS)
    if kind == "example_2d":
        return dict(kind=kind, h=side(64, 384), w=side(72, 384))
    if kind == "plume_2d":
        return dict(kind=kind, h=side(96, 1400), w=side(96, 1400), circles=rng.randrange(0, 7))
    if kind == "step_3d":
        unit = rng.choice((1, 2, 16))
        d, h, w = (side(48, 256, unit) for _ in range(3))
        return dict(kind=kind, d=d, h=h, w=w, shape=rng.choice(("open", "boxes", "sphere")))
    if kind == "batch_2d":
        return dict(kind=kind, count=side(16, 256), lo=64, hi=side(128, 512, 32), unit=rng.choice((1, 32)))
    if kind == "cg":
        precond, dtype = rng.choice(("none", "jacobi")), rng.choice(("f32", "f64"))
        if rng.random() < 0.5:
            return dict(kind=kind, d=0, h=side(96, 1024), w=side(96, 1024), precond=precond, dtype=dtype)
        d, h, w = (side(64, 192, rng.choice((1, 16))) for _ in range(3))
        return dict(kind=kind, d=d, h=h, w=w, precond=precond, dtype=dtype)
    if kind == "transport_3d":
        d, h, w = (side(48, 256) for _ in range(3))
        return dict(kind=kind, d=d, h=h, w=w, scheme=rng.randrange(3), dtype=rng.choice(("f32", "f32", "f64")))
    if kind in ("network_3d", "train_3d"):
        d, h, w = (side(32, 128 if kind == "network_3d" else 96, 4) for _ in range(3))
        return dict(kind=kind, d=d, h=h, w=w)
    levels = rng.randrange(2, 7)
    h, w = (side(256, 4096, 1 << levels) for _ in range(2))
    return dict(kind=kind, h=h, w=w, levels=levels, filter=rng.randrange(5))


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.

def _dims(case):
    return tuple(case[k] for k in ("d", "h", "w") if case.get(k))


def _dtype(case):
    return torch.float64 if case["kind"] == "example_2d" or case.get("dtype") == "f64" else torch.float32


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _smooth(a, passes=3):
    """`passes` passes of a 3-wide box filter along every axis, edges repeated."""
    pad = (1, 1) * a.dim()
    pool = torch.nn.functional.avg_pool3d if a.dim() == 3 else torch.nn.functional.avg_pool2d
    for _ in range(passes):
        a = pool(torch.nn.functional.pad(a[None, None], pad, mode="replicate"), 3, stride=1)[0, 0]
    return a


def _face_shapes(dims):
    return [tuple(n + (i == ax) for i, n in enumerate(dims)) for ax in range(len(dims))]


def _velocity(dims, gen, umax=2.0):
    """Filtered noise on the faces, closed walls, max |u| = umax; flat, in the
    package's face layout (the part normal to the slowest axis first)."""
    parts = []
    for ax, shape in enumerate(_face_shapes(dims)):
        p = _smooth(torch.randn(shape, generator=gen, device="cuda"))
        p.select(ax, 0).zero_()
        p.select(ax, dims[ax]).zero_()
        parts.append(p)
    scale = umax / torch.stack([p.abs().max() for p in parts]).max()
    return torch.cat([p.reshape(-1) for p in parts]) * scale


def _density(dims, gen):
    a = _smooth(torch.randn(dims, generator=gen, device="cuda"))
    return (a - a.min()) / (a.max() - a.min())


def _centres(dims):
    return torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float32) + 0.5 for n in dims], indexing="ij")


def _circles(dims, count, rng, rmin, rmax):
    m = torch.zeros(dims, dtype=torch.uint8, device="cuda")
    c = _centres(dims)
    for _ in range(count):
        r = rng.uniform(rmin, rmax)
        at = [rng.uniform(0, n) for n in dims]
        m |= (sum((x - a) ** 2 for x, a in zip(c, at)) < r * r).to(torch.uint8)
    return m


def _solid(case, seed):
    """Solid cells of the case (uint8), or None."""
    dims = _dims(case)
    rng = np.random.default_rng(int(seed) + 1)
    if case["kind"] == "example_2d":
        m = torch.zeros(dims, dtype=torch.uint8, device="cuda")
        h, w = dims
        y, x = h // 2 + int(rng.integers(-4, 5)), w // 3 + int(rng.integers(-4, 5))
        m[y:y + h // 8, x:x + w // 4] = 1
        return m
    if case["kind"] == "plume_2d":
        return _circles(dims, case["circles"], rng, 4, min(dims) / 8) if case["circles"] else None
    shape = case.get("shape", "boxes" if case["kind"] in ("network_3d", "train_3d") else "open")
    if shape == "open":
        return None
    if shape == "sphere":
        r = min(dims) / 8
        return (sum((x - n / 2) ** 2 for x, n in zip(_centres(dims), dims)) < r * r).to(torch.uint8)
    m = torch.zeros(dims, dtype=torch.uint8, device="cuda")
    scale = min(1.0, min(dims) / 128)
    for _ in range(int(rng.integers(1, 7))):
        size = [int(rng.integers(max(2, round(8 * scale)), max(3, round(48 * scale)) + 1)) for _ in dims]
        at = [int(rng.integers(1, max(2, n - s - 1))) for n, s in zip(dims, size)]
        m[tuple(slice(a, a + s) for a, s in zip(at, size))] = 1
    return m


def _frame(case, seed):
    """(velocity, density) of a frame, in the case's type."""
    gen, dims, dt = _generator(seed), _dims(case), _dtype(case)
    return _velocity(dims, gen).to(dt), _density(dims, gen).to(dt)


def _batch(case, seed):
    """Sides, masks, sources and fields of a batch of plumes."""
    rng, gen = np.random.default_rng(int(seed)), _generator(seed)
    sides = np.arange(case["lo"], case["hi"] + 1, case["unit"])
    sides = np.random.default_rng(case["count"]).choice(sides, (case["count"], 2))  # the same for every seed
    out = []
    for dims in map(tuple, sides.tolist()):
        m = _circles(dims, int(rng.integers(0, 9)), rng, 4, 32)
        at = [int(rng.integers(0, n)) for n in dims]
        edge = int(rng.integers(0, 4))
        at[edge & 1] = 0 if edge < 2 else dims[edge & 1] - 1
        m[tuple(slice(max(0, a - 2), a + 3) for a in at)] = 0  # the source cell stays fluid
        y, x = _centres(dims)
        src = torch.exp(-((y - 0.5 - at[0]) ** 2 + (x - 0.5 - at[1]) ** 2) / 32.0) * (m == 0)
        out.append((dims, m, src, _velocity(dims, gen), _density(dims, gen)))
    return out


CIN = (16, 16, 16, 32, 32, 64, 96, 32, 48, 16)
COUT = (16, 16, 32, 32, 64, 64, 32, 32, 16, 16)


def _net_params(seed):
    """He-normal weights in the network's layout: per layer [27][in][out]
    (layer 0 uses 2 of its 16 inputs), then the 16 output weights."""
    rng = np.random.default_rng(int(seed) + 7)
    parts = []
    for k, (ci, co) in enumerate(zip(CIN, COUT)):
        real = 2 if k == 0 else ci
        a = rng.standard_normal((27, ci, co)) * math.sqrt(2.0 / (27 * real))
        a[:, real:] = 0
        parts.append(a.ravel())
    parts.append(0.3 * rng.standard_normal(16))
    return np.concatenate(parts).astype(np.float32)


def _net_inputs(case, seed):
    """(solid, b, p): a divergence with boxes and its pressure (plain CG)."""
    dims = _dims(case)
    solid = _solid(case, seed)
    vel = _velocity(dims, _generator(seed))
    sys = _System(dims, solid, torch.float64)
    b = sys.rhs(sys.split(vel.double()))
    p, _ = sys.cg(b, 1.0, 200, 0.0)
    return solid, b[0].float(), p[0].float()


def _solver(case):
    if case["kind"] == "example_2d":
        return pg.SolverConfig()  # the reference's: plain CG, threshold 0.1, 100 iterations
    if case["kind"] == "batch_2d":
        return pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-6, max_iter=100000)
    return pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-5 if case["kind"] == "plume_2d" else 1e-6,
                           max_iter=20000, refine=4)


def _flow(case):
    """(time step, buoyancy) of a step case."""
    if case["kind"] == "example_2d":
        return 0.05, 0.0
    if case["kind"] == "step_3d" and case["shape"] == "open":
        return 1.0, 0.0
    return 0.5, 1.0


def _grid(dims, solid):
    g = pg.Grid2d(dims) if len(dims) == 2 else pg.Grid3d(dims)
    if solid is not None:
        g.set_solid_cells(solid)
    return g


# ---------------------------------------------------------------------------
# The cases.

def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "batch_2d":
        grids = _batch(case, seed)
        b = pg.Batch2d([g[0] for g in grids])
        b.set_solid_cells([g[1].cpu().numpy() for g in grids])
        dt, buoyancy = _flow(case)
        cfg = pg.StepConfig(dt=dt, buoyancy=buoyancy, source_enabled=False, walls_after_advect=True,
                            zero_solid_after_project=True, solver=_solver(case))
        s.update(batch=b, config=cfg, source=torch.cat([g[2].reshape(-1) for g in grids]),
                 vel0=torch.cat([g[3] for g in grids]), rho0=torch.cat([g[4].reshape(-1) for g in grids]),
                 vel=b.new_faces(), rho=b.new_cells(), p=b.new_cells())
        return s
    if kind == "wavelet_2d":
        s.update(case=case, field=_density((case["h"], case["w"]), _generator(seed)).double())
        s.update(coeff=torch.empty_like(s["field"]), back=torch.empty_like(s["field"]))
        return s
    dims = _dims(case)
    if kind in ("network_3d", "train_3d"):
        solid, b, p = _net_inputs(case, seed)
        g = _grid(dims, solid)
        s.update(grid=g, net=pg.PressureNet(dims, params=_net_params(seed), out_scale=2.0),
                 b=pg.Simplex2(g, b), p=pg.Simplex2(g, p), x=g.new_simplex_2())
        return s
    dtype = _dtype(case)
    g = _grid(dims, _solid(case, seed))
    vel, rho = _frame(case, seed)
    if kind == "cg":
        b = g.new_simplex_2(dtype)
        g.divergence_rhs(b, pg.Simplex1(g, vel))
        s.update(grid=g, op=pg.LaplacianOperator(g, 1.0), m=pg.JACOBI if case["precond"] == "jacobi" else pg.IDENTITY,
                 b=b, **{k: g.new_simplex_2(dtype) for k in ("x", "r", "aux", "search")})
        return s
    s.update(grid=g, vel0=pg.Simplex1(g, vel), rho0=pg.Simplex2(g, rho), vel=g.new_simplex_1(dtype),
             rho=g.new_simplex_2(dtype), scheme=case.get("scheme"))
    if kind == "transport_3d":
        return s
    dt, buoyancy = _flow(case)
    if kind == "example_2d":
        h, w = dims
        cfg = pg.StepConfig(dt=dt, source_lo=(0, 5, w // 2 - 10), source_hi=(1, 20, w // 2), solver=_solver(case))
    else:
        cfg = pg.StepConfig(dt=dt, buoyancy=buoyancy, source_enabled=False, walls_after_advect=True,
                            zero_solid_after_project=True, solver=_solver(case))
    s.update(config=cfg, p=g.new_simplex_2(dtype))
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch_2d":
        s["vel"].copy_(s["vel0"])
        s["rho"].copy_(s["rho0"])
        s["batch"].step(s["config"], s["vel"], s["rho"], s["p"], source_field=s["source"])
        return {"vel": s["vel"], "rho": s["rho"], "p": s["p"]}
    if kind == "wavelet_2d":
        c = s["case"]
        s["coeff"].copy_(s["field"])
        wavelet.fwt_2d(s["coeff"], c["levels"], c["filter"])
        s["back"].copy_(s["coeff"])
        wavelet.ifwt_2d(s["back"], c["levels"], c["filter"])
        return {"coeff": s["coeff"], "back": s["back"]}
    if kind == "network_3d":
        s["net"].forward(s["grid"], s["b"], 1.0, s["x"])
        return {"x": s["x"].data}
    if kind == "train_3d":
        s["net"].zero_grads()
        loss = s["net"].accumulate(s["grid"], s["b"], s["p"], 1.0)
        return {"loss": loss, "grad": s["net"].get_grads()}
    if kind == "cg":
        pg.precond_conjugate_gradient(s["m"], s["x"], s["b"], 100, 1e-30, s["r"], s["aux"], s["search"], s["op"])
        return {"x": s["x"].data, "r": s["r"].data}
    if kind == "transport_3d":
        pg.advect_mac(s["vel"], s["vel0"], 1.0, s["vel0"])
        if s["scheme"]:
            pg.advect2(s["rho"], s["rho0"], 1.0, s["vel0"], s["scheme"])
        else:
            pg.advect(s["rho"], s["rho0"], 1.0, s["vel0"])
        return {"vel": s["vel"].data, "rho": s["rho"].data}
    s["vel"].assign(s["vel0"])
    s["rho"].assign(s["rho0"])
    pg.step(s["grid"], s["config"], s["vel"], s["rho"], s["p"])
    return {"vel": s["vel"].data, "rho": s["rho"].data, "p": s["p"].data}


def work(case):
    """Fields read once and written once; the arithmetic of the stencils per
    cell and iteration, and of the convolutions."""
    kind = case["kind"]
    if kind == "batch_2d":
        cells = case["count"] * ((case["lo"] + case["hi"]) / 2) ** 2
        return {"bytes": cells * 33, "flops": cells * 1000}  # vel, rho, source, flags in; vel, rho, p out
    dims = _dims(case)
    cells, size = math.prod(dims), _dtype(case).itemsize
    if kind == "wavelet_2d":
        taps = wavelet.TAPS[case["filter"]]
        return {"bytes": cells * 8 * 4, "flops": cells * 4 * 2 * taps * 4 / 3}
    if kind in ("network_3d", "train_3d"):
        level = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0)
        flops = sum(2 * 27 * ci * co * cells / 8 ** lv for ci, co, lv in zip(CIN, COUT, level))
        return {"bytes": cells * 9, "flops": flops * (1 if kind == "network_3d" else 3)}
    if kind == "cg":
        return {"bytes": cells * (3 * size + 1), "flops": cells * 100 * 25}
    faces = sum(math.prod(f) for f in _face_shapes(dims))
    fields = (faces + cells) * size * 2
    if kind == "transport_3d":
        return {"bytes": fields, "flops": cells * 200}
    return {"bytes": fields + cells * (size + 1), "flops": cells * (2500 if kind == "example_2d" else 1000)}


# ---------------------------------------------------------------------------
# The same results in 64 bits, written out in plain torch.

class _System:
    """The discrete operators on a stack of grids.  Arrays have a leading
    axis over the grids; a grid smaller than the stack's shape fills its low
    corner (`sides`: its extent per axis, shape (B, 1, ...))."""

    def __init__(self, dims, solid=None, dtype=torch.float64, sides=None):
        self.dims, self.nd = dims, len(dims)
        self.B = 1 if sides is None else len(sides)
        one = (self.B,) + (1,) * self.nd
        self.n = [torch.tensor([s[a] for s in sides] if sides else [dims[a]], device="cuda").view(one)
                  for a in range(self.nd)]
        fluid = torch.ones((self.B,) + tuple(dims), dtype=torch.bool, device="cuda")
        for a in range(self.nd):
            fluid &= self.at(a, dims[a]) < self.n[a]
        self.inside = fluid
        if solid is not None:
            fluid = fluid & (solid.view(fluid.shape) == 0)
        self.open = []  # interior faces between two fluid cells
        for a in range(self.nd):
            o = torch.zeros((self.B,) + _face_shapes(dims)[a], dtype=dtype, device="cuda")
            o.narrow(a + 1, 1, dims[a] - 1).copy_(fluid.narrow(a + 1, 1, dims[a] - 1) & fluid.narrow(a + 1, 0, dims[a] - 1))
            self.open.append(o)

    def at(self, a, count):
        """Indices 0 .. count - 1 along axis a, broadcastable."""
        shape = [1] * (self.nd + 1)
        shape[a + 1] = count
        return torch.arange(count, device="cuda").view(shape)

    def split(self, flat):
        out, o = [], 0
        for shape in _face_shapes(self.dims):
            k = math.prod(shape)
            out.append(flat[o:o + k].view((1,) + shape))
            o += k
        return out

    def wall(self, a):
        i = self.at(a, self.dims[a] + 1)
        return (i == 0) | (i == self.n[a])

    def walls(self, vel):
        return [torch.where(self.wall(a), torch.zeros_like(v), v) for a, v in enumerate(vel)]

    def centred(self, vel, a):
        v, n = vel[a], self.dims[a]
        return 0.5 * (v.narrow(a + 1, 0, n) + v.narrow(a + 1, 1, n))

    def sample(self, q, corners):
        """q at per-axis (low index, high index, fraction)."""
        out = 0
        shape = torch.broadcast_shapes(*[c[2].shape for c in corners])
        flat = q.reshape(self.B, -1)
        for pick in itertools.product((0, 1), repeat=self.nd):
            index, weight = 0, 1
            for a, (k, c) in enumerate(zip(pick, corners)):
                index = index * q.shape[a + 1] + c[k]
                weight = weight * (c[2] if k else 1 - c[2])
            index = index.expand(shape).reshape(self.B, -1)
            out = out + weight * flat.gather(1, index).view(shape)
        return out

    def trace_cells(self, dt, vel):
        """Where each cell's back-trace lands: per axis (low, high, fraction)."""
        got = []
        for a in range(self.nd):
            p = self.at(a, self.dims[a]) - dt * self.centred(vel, a)
            p = torch.minimum(p.clamp(min=0), self.n[a] - 1.00001)
            i = torch.minimum(p.floor().long(), self.n[a] - 2)
            i = i.clamp(min=0)
            got.append((i, torch.minimum(i + 1, torch.tensor(self.dims[a] - 1, device="cuda")), p - i))
        return got

    def advect(self, q, dt, vel):
        return self.sample(q, self.trace_cells(dt, vel))

    def advect2(self, q, dt, vel, scheme):
        corners = self.trace_cells(dt, vel)
        q1 = self.sample(q, corners)
        q2 = self.advect(q1, -dt, vel)
        v = q1 + 0.5 * (q - q2) if scheme == 1 else self.sample(q + 0.5 * (q - q2), corners)
        picks = []
        for pick in itertools.product((0, 1), repeat=self.nd):
            index = 0
            for a, (k, c) in enumerate(zip(pick, corners)):
                index = index * q.shape[a + 1] + c[k]
            picks.append(q.reshape(self.B, -1).gather(1, index.reshape(self.B, -1)).view(q.shape))
        lo, hi = picks[0], picks[0]
        for v2 in picks[1:]:
            lo, hi = torch.minimum(lo, v2), torch.maximum(hi, v2)
        return torch.where((v < lo) | (v > hi), q1, v)

    def advect_mac(self, dt, vel):
        out = []
        for f in range(self.nd):  # the faces normal to axis f
            corners = []
            shape = (self.B,) + _face_shapes(self.dims)[f]
            for a in range(self.nd):
                if a == f:
                    v, off, count = vel[f], 0.0, self.n[f] + 1
                else:
                    c, i = self.centred(vel, a), self.at(f, self.dims[f] + 1)
                    hi = torch.minimum(i, self.n[f] - 1)
                    lo = (i - 1).clamp(min=0)
                    pick = [torch.take_along_dim(c, k.clamp(max=self.dims[f] - 1).expand(shape), f + 1) for k in (hi, lo)]
                    v, off, count = 0.5 * (pick[0] + pick[1]), 0.5, self.n[a]
                q = (self.at(a, shape[a + 1]) + off - dt * v) - off
                p = q.floor().clamp(min=0)
                last = count - 1
                i0 = torch.minimum(p.long(), last)
                corners.append((i0, torch.minimum(i0 + 1, last), (q - p).clamp(0, 1)))
            out.append(self.sample(vel[f], corners))
        return out

    def rhs(self, vel):
        b = 0
        for a, v in enumerate(vel):
            v = torch.where((self.open[a] > 0) | self.wall(a), v, torch.zeros_like(v))
            b = b - (v.narrow(a + 1, 1, self.dims[a]) - v.narrow(a + 1, 0, self.dims[a]))
        return torch.where(self.inside, b, torch.zeros_like(b))

    def laplacian(self, p, dt):
        out = torch.zeros_like(p)
        for a in range(self.nd):
            n = self.dims[a]
            g = (p.narrow(a + 1, 1, n - 1) - p.narrow(a + 1, 0, n - 1)) * self.open[a].narrow(a + 1, 1, n - 1)
            out.narrow(a + 1, 1, n - 1).add_(g, alpha=dt)
            out.narrow(a + 1, 0, n - 1).sub_(g, alpha=dt)
        return out

    def cg(self, b, dt, iterations, threshold, jacobi=False, rel=0.0):
        """Conjugate gradient; stops where every grid's largest residual is
        below `threshold`, or below `rel` of its largest right-hand side
        (looked at every 20 iterations)."""
        axes = tuple(range(1, self.nd + 1))
        inv = 1.0
        if jacobi:
            k = sum(o.narrow(a + 1, 0, self.dims[a]) + o.narrow(a + 1, 1, self.dims[a]) for a, o in enumerate(self.open))
            inv = torch.where(k > 0, 1 / (k * dt).clamp(min=1e-30), torch.zeros_like(k))
        x, r = torch.zeros_like(b), b.clone()
        stop = rel * b.abs().amax(axes, keepdim=True)
        if threshold and float(b.abs().max()) < threshold:
            return x, r
        z = r * inv
        p, sigma = z.clone(), (z * r).sum(axes, keepdim=True)
        for k in range(iterations):
            ap = self.laplacian(p, dt)
            pap = (p * ap).sum(axes, keepdim=True)
            alpha = torch.where(pap > 0, sigma / pap, torch.zeros_like(pap))
            x += alpha * p
            r -= alpha * ap
            if threshold and float(r.abs().max()) < threshold:
                break
            if rel and k % 20 == 19 and bool((r.abs().amax(axes, keepdim=True) <= stop).all()):
                break
            z = r * inv
            new = (z * r).sum(axes, keepdim=True)
            p.mul_(torch.where(sigma > 0, new / sigma, torch.zeros_like(new))).add_(z)
            sigma = new
        return x, r

    def project(self, vel, p, dt, zero_solid):
        out = []
        for a, v in enumerate(vel):
            n = self.dims[a]
            v = v.clone()
            v.narrow(a + 1, 1, n - 1).sub_(p.narrow(a + 1, 1, n - 1) - p.narrow(a + 1, 0, n - 1), alpha=dt)
            out.append(v * self.open[a] if zero_solid else v)
        return self.walls(out)


def _exact_step(sys, vel, rho, dt, buoyancy):
    """A closed-wall step, the pressure solved far below any tolerance."""
    new = sys.advect(rho, dt, vel)
    vel = sys.walls(sys.advect_mac(dt, vel))
    y = sys.nd - 2
    n = sys.dims[y]
    if buoyancy:
        lift = 0.5 * (new.narrow(y + 1, 1, n - 1) + new.narrow(y + 1, 0, n - 1))
        vy = vel[y].clone()
        vy.narrow(y + 1, 1, n - 1).add_(lift, alpha=dt * buoyancy)
        vel[y] = torch.where(sys.wall(y), torch.zeros_like(vy), vy)
    p, _ = sys.cg(sys.rhs(vel), dt, 6000, 0.0, jacobi=True, rel=1e-11)
    return sys.project(vel, p, dt, True), new


def _exact_net(case, seed):
    """The network in 64 bits: its output, or its loss and gradients."""
    dims = _dims(case)
    solid, b, p_true = _net_inputs(case, seed)
    sys = _System(dims, solid)
    b, p_true = b.double(), p_true.double()
    faces = sum(o.narrow(a + 1, 0, dims[a]) + o.narrow(a + 1, 1, dims[a]) for a, o in enumerate(sys.open))[0]
    theta = torch.from_numpy(_net_params(seed)).cuda().double().requires_grad_(case["kind"] == "train_3d")
    s, m = b.square().mean().sqrt(), faces > 0
    o = 0

    def layer(k, x):  # x: (channels, d, h, w); 27 shifted products
        nonlocal o
        wk = theta[o:o + 27 * CIN[k] * COUT[k]].view(27, CIN[k], COUT[k])
        o += wk.numel()
        if k == 0:
            wk = wk[:, :2]
        size = x.shape[1:]
        x = torch.nn.functional.pad(x, (1, 1) * 3)
        y = 0
        for t in range(27):
            part = x[:, t // 9:t // 9 + size[0], t // 3 % 3:t // 3 % 3 + size[1], t % 3:t % 3 + size[2]]
            y = y + torch.einsum("io,idhw->odhw", wk[t], part)
        return torch.relu(y)

    def pool(x):
        return torch.nn.functional.avg_pool3d(x[None], 2)[0]

    def up(x):
        for a in (1, 2, 3):
            x = x.repeat_interleave(2, a)
        return x

    y1 = layer(1, layer(0, torch.stack([b / s, faces / 6])))
    y3 = layer(3, layer(2, pool(y1)))
    y5 = layer(5, layer(4, pool(y3)))
    y7 = layer(7, layer(6, torch.cat([up(y5), y3])))
    y9 = layer(9, layer(8, torch.cat([up(y7), y1])))
    q = torch.einsum("c,cdhw->dhw", theta[o:], y9) * m
    if case["kind"] == "network_3d":
        return {"x": q * s * 2.0}
    e = (q - p_true / (s * 2.0)) * m
    jump = [(e.narrow(a, 1, n - 1) - e.narrow(a, 0, n - 1)).square() * sys.open[a][0].narrow(a, 1, n - 1)
            for a, n in enumerate(dims)]
    loss = sum(j.sum() for j in jump) / e.numel()
    loss.backward()
    grad = theta.grad.clone()
    grad[:27 * 16 * 16].view(27, 16, 16)[:, 2:] = 0  # inputs that are always zero
    return {"loss": loss.detach(), "grad": grad.cpu().numpy()}


def _filters(kind):
    """(analysis low, analysis high, synthesis low, synthesis high): the
    published Haar and biorthogonal spline coefficients."""
    r = math.sqrt(0.5)
    low = {  # analysis low, synthesis low; the high filters alternate their signs
        wavelet.HAAR: ([1, 1], [1, 1]),
        wavelet.BIOR13: ([-1 / 8, 1 / 8, 1, 1, 1 / 8, -1 / 8], [0, 0, 1, 1, 0, 0]),
        wavelet.BIOR22: ([0, -1 / 4, 1 / 2, 3 / 2, 1 / 2, -1 / 4], [0, 1 / 2, 1, 1 / 2, 0, 0]),
        wavelet.BIOR24: ([0, 3 / 64, -3 / 32, -1 / 4, 19 / 32, 45 / 32, 19 / 32, -1 / 4, -3 / 32, 3 / 64],
                         [0, 0, 0, 1 / 2, 1, 1 / 2, 0, 0, 0, 0]),
        wavelet.BIOR31: ([-1 / 2, 3 / 2, 3 / 2, -1 / 2], [1 / 4, 3 / 4, 3 / 4, 1 / 4]),
    }[kind]
    dl, ul = ([r * v for v in f] for f in low)
    dh = [(-1) ** (k + 1) * v for k, v in enumerate(ul)]
    uh = [(-1) ** k * v for k, v in enumerate(dl)]
    return dl, dh, ul, uh


def _exact_wavelet(case, seed):
    """fwt_2d / ifwt_2d as gathers and scatters along one axis at a time."""
    dl, dh, ul, uh = _filters(case["filter"])
    n = len(dl)

    def down(a):  # along the last axis, mirrored samples
        size = a.shape[-1]
        i = torch.arange(size // 2, device="cuda")
        low = high = 0
        for f in range(n):
            k = 2 * i + f - n // 2 + 1
            k = torch.where(k < 0, -k, torch.where(k >= size, size - 1 - k % size, k))
            low = low + a[..., k] * dl[n - 1 - f]
            high = high + a[..., k] * dh[n - 1 - f]
        return torch.cat([low, high], -1)

    def up(a):  # wrapped scatter
        size = a.shape[-1]
        i = torch.arange(size // 2, device="cuda")
        out = torch.zeros_like(a)
        for f in range(n):
            out.index_add_(a.dim() - 1, (2 * i + f - n // 2 + 1) % size,
                           a[..., :size // 2] * ul[f] + a[..., size // 2:] * uh[f])
        return out

    a = _density((case["h"], case["w"]), _generator(seed)).double()
    shapes = [(case["h"] >> k, case["w"] >> k) for k in range(case["levels"])]
    for r, c in shapes:
        a[:r, :c] = down(a[:r, :c])
        a[:r, :c] = down(a[:r, :c].T).T
    coeff = a.clone()
    for r, c in reversed(shapes):
        a[:r, :c] = up(a[:r, :c].T.contiguous()).T
        a[:r, :c] = up(a[:r, :c].contiguous())
    return {"coeff": coeff, "back": a}


def exact(case, seed):
    kind = case["kind"]
    if kind == "wavelet_2d":
        return _exact_wavelet(case, seed)
    if kind in ("network_3d", "train_3d"):
        return _exact_net(case, seed)
    if kind == "batch_2d":
        if case["count"] * case["hi"] ** 2 > 40e6:
            return None
        grids = _batch(case, seed)
        dims = tuple(max(g[0][a] for g in grids) for a in (0, 1))

        def stack(parts, shape):
            out = torch.zeros((len(parts),) + shape, dtype=torch.float64, device="cuda")
            for o, p in zip(out, parts):
                o[:p.shape[0], :p.shape[1]] = p
            return out

        sys = _System(dims, stack([g[1] for g in grids], dims), sides=[g[0] for g in grids])
        parts = [_System(g[0]).split(g[3].double()) for g in grids]
        vel = [stack([p[a][0] for p in parts], _face_shapes(dims)[a]) for a in (0, 1)]
        rho = torch.maximum(stack([g[4] for g in grids], dims), stack([g[2] for g in grids], dims))
        vel, rho = _exact_step(sys, vel, rho, *_flow(case))
        flat = []
        for i, g in enumerate(grids):
            flat += [vel[a][i][:s[0], :s[1]].reshape(-1) for a, s in enumerate(_face_shapes(g[0]))]
        return {"vel": torch.cat(flat), "p": None,
                "rho": torch.cat([rho[i][:g[0][0], :g[0][1]].reshape(-1) for i, g in enumerate(grids)])}
    dims = _dims(case)
    if math.prod(dims) > 20e6:
        return None
    sys = _System(dims, _solid(case, seed))
    vel, rho = _frame(case, seed)
    vel, rho = sys.split(vel.double()), rho.double()[None]
    if kind == "cg":
        x, r = sys.cg(sys.rhs(vel), 1.0, 100, 0.0, jacobi=case["precond"] == "jacobi")
        return {"x": x[0], "r": r[0]}
    if kind == "transport_3d":
        new = sys.advect2(rho, 1.0, vel, case["scheme"]) if case["scheme"] else sys.advect(rho, 1.0, vel)
        return {"vel": torch.cat([v.reshape(-1) for v in sys.advect_mac(1.0, vel)]), "rho": new[0]}
    dt, buoyancy = _flow(case)
    if kind == "example_2d":
        w = dims[1]
        rho, vel = rho.clone(), [v.clone() for v in vel]
        rho[:, 5:20, w // 2 - 10:w // 2] = 1.0
        vel[0][:, 5:20, w // 2 - 10:w // 2] = 20.0
        new = sys.advect(rho, dt, vel)
        vel = sys.advect_mac(dt, vel)
        p, _ = sys.cg(sys.rhs(vel), dt, 100, 0.1)
        return {"vel": torch.cat([v.reshape(-1) for v in sys.project(vel, p, dt, False)]), "rho": new[0], "p": p[0]}
    vel, rho = _exact_step(sys, vel, rho, dt, buoyancy)
    return {"vel": torch.cat([v.reshape(-1) for v in vel]), "rho": rho[0], "p": None}
