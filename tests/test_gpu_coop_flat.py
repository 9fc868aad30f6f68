"""The cooperative CG on flat double grids, whose halos are larger than their
blocks' cells, and on the ones that its rule leaves to the loop: the loop's
results, and the kernel that the rule names did the work."""
import pytest

import test_gpu_coop as coop

pytestmark = pytest.mark.gpu

TAKEN = [(4, 64, 64), (8, 50, 50), (3, 20, 20), (12, 100, 100), (10, 3000), (40, 2000)]
LEFT = [(8, 100, 100), (2, 85, 85), (10, 8000)]


@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("dims", TAKEN + LEFT)
def test_flat_grids_agree(pg, oracle, dims, precond, monkeypatch):
    coop.test_double_solves_agree(pg, oracle, dims, precond, monkeypatch)


@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("dims", TAKEN + LEFT + [(128, 128), (64, 64, 64), (900, 900)])
def test_route(pg, oracle, dims, precond):
    """Launches of a 40-iteration solve: two per iteration in the loop."""
    lib = pg.load()
    g, b = coop.problem(pg, oracle, dims)
    coop.solve(pg, g, b, precond, 40, 1e-300)
    before = lib.pg_kernel_launches()
    st, _ = coop.solve(pg, g, b, precond, 40, 1e-300)
    n = lib.pg_kernel_launches() - before
    assert st["iterations"] == 40
    taken = dims in TAKEN or dims in [(128, 128), (64, 64, 64)]
    assert n < 10 if taken else n >= 80, (dims, n)
