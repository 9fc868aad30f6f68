"""The marching multigrid kernels of a batch (strips of 64 columns, rows in
pairs, the shared-memory tail) against an FP64 MG-PCG in numpy, at widths
around the strips' edges and overlaps, odd widths and heights, chunks' last
rows, grids that the tail takes whole, thin ones, and pockets."""
import numpy as np
import pytest
import torch

from conftest import rng

pytestmark = pytest.mark.gpu

DIMS = [(64, 64), (65, 63), (70, 80), (90, 65), (33, 119), (97, 120), (40, 121), (130, 176), (129, 177), (257, 301),
        (600, 66), (3, 800), (5, 1300), (2, 900), (8, 8), (9, 7), (13, 5), (1023, 58), (48, 60), (66, 124)]
DT = 0.5


class Level:
    """Weights of a level: wx[y, x] of the face left of the cell, wy above it."""

    def __init__(self, wx, wy):
        self.wx, self.wy, (self.h, self.w) = wx, wy, wx.shape
        self.wr = np.pad(wx, ((0, 0), (0, 1)))[:, 1:]
        self.wd = np.pad(wy, ((0, 1), (0, 0)))[1:]
        diag = wx + self.wr + wy + self.wd
        self.inv = np.divide(1.0, diag, out=np.zeros_like(diag), where=diag > 0)
        self.diag = diag
        y, x = np.indices(wx.shape)
        self.colour = (x + y) & 1

    def around(self, e):
        p = np.pad(e, 1)
        return self.wx * p[1:-1, :-2] + self.wr * p[1:-1, 2:] + self.wy * p[:-2, 1:-1] + self.wd * p[2:, 1:-1]

    def half(self, e, f, colour):
        return np.where(self.colour == colour, (f + self.around(e)) * self.inv, e)

    def residual(self, e, f):
        return f - (self.diag * e - self.around(e))

    def coarser(self):
        def pad(a):
            return np.pad(a, ((0, self.h & 1), (0, self.w & 1)))

        wx, wy = pad(self.wx), pad(self.wy)
        return Level(0.5 * (wx[0::2, 0::2] + wx[1::2, 0::2]), 0.5 * (wy[0::2, 0::2] + wy[0::2, 1::2]))

    def restrict(self, r):
        r = np.pad(r, ((0, self.h & 1), (0, self.w & 1)))
        return r[0::2, 0::2] + r[1::2, 0::2] + r[0::2, 1::2] + r[1::2, 1::2]


def vcycle(levels, f, ns):
    L = levels[0]
    e = np.zeros_like(f)
    if len(levels) == 1:
        s = max(L.h, L.w)
        pairs = min(32, max(4, (s * s + 1) // 2))
        for order in ((0, 1), (1, 0)):
            for _ in range(pairs):
                for c in order:
                    e = L.half(e, f, c)
        return e
    for _ in range(ns):
        e = L.half(L.half(e, f, 0), f, 1)
    c = vcycle(levels[1:], L.restrict(L.residual(e, f)), ns)
    e = e + np.repeat(np.repeat(c, 2, 0), 2, 1)[:L.h, :L.w]
    for _ in range(ns):
        e = L.half(L.half(e, f, 1), f, 0)
    return e


def solve(mask, b, iters, ns, lab, n):
    fluid = mask == 0
    wx, wy = np.zeros(mask.shape), np.zeros(mask.shape)
    wx[:, 1:] = DT * (fluid[:, 1:] & fluid[:, :-1])
    wy[1:] = DT * (fluid[1:] & fluid[:-1])
    levels = [Level(wx, wy)]
    while min(levels[-1].h, levels[-1].w) > 2 and levels[-1].h * levels[-1].w > 64:
        levels.append(levels[-1].coarser())

    def project(a):
        a = a.copy()
        for k in range(1, n + 1):
            a[lab == k] -= a[lab == k].mean()
        return a

    A = levels[0]
    r = project(b)
    z = project(vcycle(levels, r, ns))
    x, p, sigma = np.zeros_like(b), z, (z * r).sum()
    for _ in range(iters):
        ap = A.diag * p - A.around(p)
        alpha = sigma / (p * ap).sum()
        x, r = x + alpha * p, project(r - alpha * ap)
        z = project(vcycle(levels, r, ns))
        s = (z * r).sum()
        p, sigma = z + s / sigma * p, s
    return x


@pytest.mark.parametrize("nsmooth", [1, 2, 3])
@pytest.mark.parametrize("iters", [1, 3])
def test_solve_matches_fp64(pg, oracle, nsmooth, iters):
    """p after a few iterations.  A V-cycle's FP32 sweeps keep an error of a few
    roundings (6e-8) per level and damp what they get, the coarsest level's 128
    half-sweeps add sqrt(128) of them to its smoothest mode, sums move alpha
    and beta by an ulp: 1e-5 of max |p| per component leaves a factor of 10."""
    from panopaea_gb300 import workloads as W
    from scipy import ndimage

    r = rng(5)
    masks, vels = [], []
    for i, (h, w) in enumerate(DIMS):
        m = np.zeros((h, w), np.uint8)
        if i % 3 == 1 and min(h, w) > 12:
            m[h // 3:h // 3 + 5, w // 3:w // 3 + 5] = 1
        if i % 3 == 2 and min(h, w) > 30:  # a box with a pocket inside
            m[h // 2:h // 2 + 9, w // 2:w // 2 + 9] = 1
            m[h // 2 + 2:h // 2 + 7, w // 2 + 2:w // 2 + 7] = 0
        masks.append(m)
        parts = [r.standard_normal(s).astype(np.float32) for s in W.face_shapes((h, w))]
        W.zero_walls(parts)
        vels.append(np.concatenate([p.ravel() for p in parts]))
    B = pg.Batch2d(DIMS)
    B.set_solid_cells(masks)

    def run(max_iter):
        v = torch.from_numpy(B.pack_faces(vels)).cuda()
        rho, p = B.new_cells(), B.new_cells()
        cfg = pg.StepConfig(dt=DT, source_enabled=False, walls_after_advect=True, zero_solid_after_project=True,
                            solver=pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-30, max_iter=max_iter,
                                                   mg_smooth=nsmooth))
        return v, p, B.step(cfg, v, rho, p)

    v0, _, _ = run(0)  # the advected velocity: nothing is projected
    _, p, stats = run(iters)
    for i, (h, w) in enumerate(DIMS):
        assert stats[i]["iterations"] == iters
        lab, n = ndimage.label(masks[i] == 0)
        vel = B.faces_of(v0, i).cpu().numpy().astype(np.float64)
        b = oracle.divergence_rhs(vel, (h, w), oracle.cell_mask_to_faces(masks[i])).reshape(h, w)
        want = solve(masks[i], b, iters, nsmooth, lab, n)
        got = B.cells_of(p, i).cpu().numpy().astype(np.float64).reshape(h, w)
        for k in range(1, n + 1):
            x, y = got[lab == k], want[lab == k]
            x, y = x - x.mean(), y - y.mean()
            assert np.abs(x - y).max() <= 1e-5 * np.abs(want).max(), (i, h, w, k)
