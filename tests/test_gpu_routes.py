"""The multigrid kernels that the comparisons with the diagnostic switches mean
to compare are the ones that run: a comparison whose fast path has declined
compares a path with itself.  And the fused pairs with two and three sweeps
(one sweep has no plain pair), on the shapes of test_gpu_pair_columns.py."""
import numpy as np
import pytest

import test_gpu_mg as mg
from conftest import rng, seed_of
from test_gpu_ops import cells, make_grid

pytestmark = pytest.mark.gpu


def sweeps(pg, dims, kind, on, monkeypatch):
    """Launches of a kind in a multigrid solve of a few iterations."""
    monkeypatch.setenv("PG_MG_CTAIL", on)
    g = make_grid(pg, dims)
    b = rng(seed_of(dims, "routes")).standard_normal(dims).astype(np.float32)
    b, x = cells(pg, g, b - b.mean()), g.new_simplex_2()
    cfg = pg.SolverConfig(precond=2, rel_stop=True, rel_tol=1e-3, max_iter=50, refine=0)
    st, n = mg._launches(pg.load(), lambda: pg.solve_pressure(g, x, b, 0.5, cfg), kind)
    assert st["status"] == 0
    return n


@pytest.mark.parametrize("dims", [(256, 256), (97, 131), (128, 64), (65, 64), (33, 400), (255, 63)])
def test_whole_2d_vcycles_are_the_tail(pg, dims, monkeypatch):
    assert sweeps(pg, dims, "mg_smooth", "1", monkeypatch) == 0
    assert sweeps(pg, dims, "mg_smooth", "0", monkeypatch) > 0


@pytest.mark.parametrize("dims", [(93, 59, 75), (66, 70, 63), (300, 281), (700, 130), (90, 901)])
def test_tails_below_the_fine_level_take_levels(pg, dims, monkeypatch):
    on, off = (sweeps(pg, dims, "mg_smooth_coarse", s, monkeypatch) for s in "10")
    assert on < off, (on, off)


@pytest.mark.parametrize("nsmooth", [2, 3])
@pytest.mark.parametrize("dims", [(40, 16, 64), (9, 33, 208), (150, 72, 160), (64, 176, 320)])
def test_plain_pairs_by_columns(pg, oracle, dims, nsmooth, monkeypatch):
    mg.test_fused_pairs_equal_half_sweeps(pg, oracle, dims, nsmooth, monkeypatch)
