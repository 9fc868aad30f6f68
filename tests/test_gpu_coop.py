"""The cooperative CG (small double grids) against the two-kernel loop on the same
grids: one block and all of them, rows longer than a block's cells, cells
that fill no warp, obstacles, both preconditioners, every way a
solve ends."""
import numpy as np
import pytest
import torch

from conftest import rng, seed_of
from test_gpu_ops import faces, host, make_grid

pytestmark = pytest.mark.gpu


def problem(pg, oracle, dims):
    r = rng(seed_of(dims, "coop"))
    vel = oracle.walls(r.standard_normal(oracle.num_faces(dims)).astype(np.float64), dims)
    g = make_grid(pg, dims)
    cs = (r.random(dims) < 0.05).astype(np.uint8)
    g.set_solid_cells(cs)
    b = g.new_simplex_2(torch.float64)
    g.divergence_rhs(b, faces(pg, g, vel))
    return g, b


def solve(pg, g, b, precond, iterations, threshold):
    v = [g.new_simplex_2(b.data.dtype) for _ in range(4)]
    m = pg.JACOBI if precond else pg.IDENTITY
    st = pg.precond_conjugate_gradient(m, v[0], b, iterations, threshold, v[1], v[2], v[3], pg.LaplacianOperator(g, 0.5))
    return st, [host(a) for a in v]


DIMS = [(1, 3), (5, 7), (64, 64), (128, 128), (33, 901), (700, 61), (257, 255), (384, 380), (9, 20, 31), (64, 64, 64), (33, 47, 50)]


@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("dims", DIMS + [(700, 800)])
def test_double_solves_agree(pg, oracle, dims, precond, monkeypatch):
    """x to 1e-10 of its largest value, r, A p and p to 1e-10 of the largest
    right-hand side (they shrink to nothing as a small grid converges, and
    their rounding errors are those of the values they came from): FP64 sums
    in two orders, 1e-15 relative, through 40 iterations."""
    g, b = problem(pg, oracle, dims)
    got = {}
    for on in ("1", "0"):
        monkeypatch.setenv("PG_CG_COOP", on)
        got[on] = solve(pg, g, b, precond, 40, 1e-9)
    (s1, v1), (s0, v0) = got["1"], got["0"]
    assert (s1["status"], s1["iterations"]) == (s0["status"], s0["iterations"])
    for k, (a, c) in enumerate(zip(v1, v0)):
        scale = np.abs(c).max() if k == 0 else np.abs(host(b)).max()
        assert np.abs(a - c).max() <= 1e-10 * max(scale, 1e-300), k


def test_ends(pg, oracle, monkeypatch):
    """b below the threshold, no iterations allowed, NaN in b, and a wait
    that gives up: the loop's statuses."""
    from panopaea_gb300 import _native as N

    lib = N.load()
    g, b = problem(pg, oracle, (90, 110))
    st, (x, r, _, _) = solve(pg, g, b, 0, 40, 1e9)
    assert st["status"] == 0 and st["iterations"] == 0 and not x.any() and np.array_equal(r, host(b))
    st, _ = solve(pg, g, b, 0, 0, 1e-9)
    assert st["status"] == N.PG_NOT_CONVERGED and st["iterations"] == 0
    default = lib.pg_debug_stage_wait_polls_default()
    assert lib.pg_debug_set_stage_wait_polls(0) == N.PG_OK
    try:
        with pytest.raises(N.PgError) as e:
            solve(pg, g, b, 0, 40, 1e-9)
        assert e.value.status == N.PG_TIMEOUT
    finally:
        assert lib.pg_debug_set_stage_wait_polls(default) == N.PG_OK
    st, _ = solve(pg, g, b, 0, 20000, 1e-9)
    assert st["status"] == 0
    b.data.view(-1)[77] = float("nan")
    with pytest.raises(N.PgError) as e:
        solve(pg, g, b, 1, 40, 1e-9)
    assert e.value.status == N.PG_NAN_DETECTED
