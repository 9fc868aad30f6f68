"""The marching pairs of a single 2D grid's levels (above the cluster tail)
against an FP64 MG-PCG in numpy whose coarsest level is solved exactly, at
sizes whose strips and rows are cut everywhere, odd rows (no pairs of
values), obstacles and a pocket."""
import numpy as np
import pytest

from conftest import rng
from test_gpu_batch_march import Level
from test_gpu_ops import faces, host, make_grid

pytestmark = pytest.mark.gpu

DT = 0.5


def vcycle(levels, pinv, f, ns):
    L = levels[0]
    if len(levels) == 1:
        return (pinv @ f.ravel()).reshape(f.shape)
    e = np.zeros_like(f)
    for _ in range(ns):
        e = L.half(L.half(e, f, 0), f, 1)
    c = vcycle(levels[1:], pinv, L.restrict(L.residual(e, f)), ns)
    e = e + np.repeat(np.repeat(c, 2, 0), 2, 1)[:L.h, :L.w]
    for _ in range(ns):
        e = L.half(L.half(e, f, 1), f, 0)
    return e


def weights(mask):
    fluid = mask == 0
    wx, wy = np.zeros(mask.shape), np.zeros(mask.shape)
    wx[:, 1:] = DT * (fluid[:, 1:] & fluid[:, :-1])
    wy[1:] = DT * (fluid[1:] & fluid[:-1])
    return wx, wy


def solve(mask, b, iters, ns, lab, n):
    levels = [Level(*weights(mask))]
    while min(levels[-1].h, levels[-1].w) > 2 and levels[-1].h * levels[-1].w > 64:
        levels.append(levels[-1].coarser())
    C = levels[-1]
    eye = np.eye(C.h * C.w).reshape(-1, C.h, C.w)
    pinv = np.linalg.pinv(np.stack([(C.diag * u - C.around(u)).ravel() for u in eye]), rcond=1e-10, hermitian=True)

    def project(a):
        a = a.copy()
        for k in range(1, n + 1):
            a[lab == k] -= a[lab == k].mean()
        return a

    A = levels[0]
    r = project(b)
    z = project(vcycle(levels, pinv, r, ns))
    x, p, sigma = np.zeros_like(b), z, (z * r).sum()
    for _ in range(iters):
        ap = A.diag * p - A.around(p)
        alpha = sigma / (p * ap).sum()
        x, r = x + alpha * p, project(r - alpha * ap)
        z = project(vcycle(levels, pinv, r, ns))
        s = (z * r).sum()
        p, sigma = z + s / sigma * p, s
    return x


@pytest.mark.parametrize("dims", [(257, 301), (264, 312), (300, 1200), (1031, 518), (130, 1999), (640, 121)])
@pytest.mark.parametrize("nsmooth", [1, 2, 3])
def test_solve_matches_fp64(pg, oracle, dims, nsmooth):
    """x after three iterations, by what its difference leaves of the operator:
    smooth differences (FP32 coarse corrections, alpha and beta an ulp apart)
    grow with the grid's sides, A of them doesn't.  The sweeps' roundings stay
    within 1e-5 of max |b|; x, stored in FP32 and added to three times, is off
    by 3 halves of an ulp per cell, which A (8 terms of weight dt) turns into
    at most 16 ulps dt max |x|."""
    from scipy import ndimage

    h, w = dims
    r = rng(h + w)
    m = np.zeros(dims, np.uint8)
    m[h // 3:h // 3 + 21, w // 3:w // 3 + 30] = 1
    if w % 2:
        m[h // 3 + 6:h // 3 + 12, w // 3 + 5:w // 3 + 14] = 0  # a pocket
    g = make_grid(pg, dims)
    g.set_solid_cells(m)
    vel = oracle.walls(r.standard_normal(oracle.num_faces(dims)).astype(np.float32), dims)
    b, x = g.new_simplex_2(), g.new_simplex_2()
    g.divergence_rhs(b, faces(pg, g, vel))
    st = pg.solve_pressure(g, x, b, DT, pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-30, max_iter=3,
                                                        mg_smooth=nsmooth))
    assert st["iterations"] == 3
    lab, n = ndimage.label(m == 0)
    want = solve(m, host(b).astype(np.float64).reshape(dims), 3, nsmooth, lab, n)
    got = host(x).astype(np.float64).reshape(dims)
    bh = host(b).astype(np.float64).reshape(dims)
    diff = np.where(m == 0, got - want, 0.0)
    A = Level(*weights(m))
    left = np.abs(A.diag * diff - A.around(diff)).max()
    assert left <= 1e-5 * np.abs(bh).max() + 16 * 2.0 ** -24 * DT * np.abs(want).max(), left
