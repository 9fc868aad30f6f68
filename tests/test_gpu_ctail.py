"""The cluster tail on the shapes where its slabs can go wrong: odd rows and
planes, ranks left without a plane, levels just above the rank-0 size, 2D
hierarchies whose tail starts below the fine level and 2D ones that it takes
in whole."""
import numpy as np
import pytest

from conftest import rng, seed_of
from test_gpu_mg import make_grid
from test_gpu_ops import faces, host

pytestmark = pytest.mark.gpu


def solve_both(pg, oracle, dims, nsmooth, monkeypatch):
    r = rng(seed_of(dims, nsmooth, "ctail2"))
    idx = np.indices(dims).astype(np.float64)
    ctr = np.array([(n - 1) / 2 for n in dims]).reshape((-1,) + (1,) * len(dims))
    cs = (((idx - ctr) ** 2).sum(0) < (min(dims) / 5.0) ** 2).astype(np.uint8)
    vel = oracle.walls(r.standard_normal(oracle.num_faces(dims)).astype(np.float32), dims)
    res = {}
    for on in ("1", "0"):
        monkeypatch.setenv("PG_MG_CTAIL", on)
        g = make_grid(pg, dims)
        g.set_solid_cells(cs)
        b = g.new_simplex_2()
        g.divergence_rhs(b, faces(pg, g, vel))
        x = g.new_simplex_2()
        cfg = pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-6, max_iter=2000, refine=4, mg_smooth=nsmooth)
        st = pg.solve_pressure(g, x, b, 0.5, cfg)
        assert st["status"] == 0 and st["true_residual_max"] <= 1e-6 * st["b_max"], (on, st)
        res[on] = (st, host(x))
    return res["1"], res["0"]


@pytest.mark.parametrize("nsmooth", [1, 2])
@pytest.mark.parametrize("dims", [(93, 59, 75), (64, 33, 17), (30, 32, 34), (66, 70, 63), (300, 281), (700, 130), (90, 901)])
def test_tail_below_the_fine_level_is_bit_identical(pg, oracle, dims, nsmooth, monkeypatch):
    (s1, x1), (s0, x0) = solve_both(pg, oracle, dims, nsmooth, monkeypatch)
    assert s1["iterations"] == s0["iterations"]
    assert np.array_equal(x1, x0)


@pytest.mark.parametrize("nsmooth", [1, 2, 3])
@pytest.mark.parametrize("dims", [(256, 256), (97, 131), (128, 64), (65, 64), (33, 400), (255, 63)])
def test_whole_2d_vcycle(pg, oracle, dims, nsmooth, monkeypatch):
    """The whole V-cycle in the cluster: the same cells' values, only z.r and
    sum(z) folded in another order, an FP64-class sum of FP32 products -- so
    beta moves by a few ulp of FP32 at most, and the solves, each to a true
    residual of 1e-6, agree to 1e-5 of the largest value up to a constant."""
    (s1, x1), (s0, x0) = solve_both(pg, oracle, dims, nsmooth, monkeypatch)
    assert abs(s1["iterations"] - s0["iterations"]) <= 1
    d = (x1 - x0).astype(np.float64)
    assert np.abs(d - np.median(d)).max() <= 1e-5 * np.abs(x0).max()
