"""Which kernels a multigrid solve takes, and in how many blocks (host code,
runtime faked; 152 SMs, three blocks on each where shared memory allows)."""
import pytest

from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
fake.fake_set_resident(3)
result = []
for dims, nsmooth in %r:
    g, x, b, st = grid(dims), cells(dims), cells(dims), N.PcgStats()
    p = solver(precond=2, refine=0, mg_smooth=nsmooth)
    log()
    rc = lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st))
    result.append((dims, nsmooth, rc, [l for l in log() if "k_mg_" in l[0]]))
    lib.pg_grid_destroy(g)
    keep.clear()
"""

# the shapes of tests/test_gpu_ctail.py, and grids too small to have a level
# above the ones that live in one block
WHOLE = [(256, 256), (97, 131), (128, 64), (65, 64), (33, 400), (255, 63)]
BELOW = [(93, 59, 75), (64, 33, 17), (30, 32, 34), (66, 70, 63), (300, 281), (700, 130), (90, 901)]
NONE = [(40, 40), (9, 70), (8, 8, 9), (20, 10, 10)]


def named(launches, *names):
    return [l for l in launches if any(n in l[0] for n in names)]


@pytest.mark.parametrize("kind", ["whole", "below", "none"])
def test_cluster_tail(host_cuda, kind):  # noqa: F811
    shapes = [(d, n) for d in {"whole": WHOLE, "below": BELOW, "none": NONE}[kind] for n in (1, 2)]
    on = host_cuda(SCRIPT % shapes)
    off = host_cuda(SCRIPT % shapes, PG_MG_CTAIL="0")
    for (dims, _, rc, a), (_, _, rc0, b) in zip(on, off):
        assert rc == 0 and rc0 == 0 and not named(b, "k_mg_ctail"), dims
        assert bool(named(a, "k_mg_ctail")) == (kind != "none"), dims
        sweeps = len(named(a, "k_mg_smooth", "k_mg_march", "k_mg_pair"))
        if kind == "whole":  # the V-cycle is the tail
            assert sweeps == 0, (dims, sweeps)
        if kind == "below":
            assert 0 < sweeps <= len(named(b, "k_mg_smooth", "k_mg_march", "k_mg_pair")), dims


def test_pairs_by_columns(host_cuda):  # noqa: F811
    """The shapes of tests/test_gpu_pair_columns.py: two whose columns of tiles
    get a whole number of blocks each, two whose blocks don't divide."""
    columns = {(40, 16, 64): 1, (9, 33, 208): 4 * 3, (150, 72, 160): 3 * 5, (64, 176, 320): 5 * 11}
    whole = {(40, 16, 64), (150, 72, 160)}
    for dims, nsmooth, rc, launches in host_cuda(SCRIPT % [(d, n) for d in columns for n in (1, 2)]):
        dims = tuple(dims)
        # template arguments: the first half-sweep's kind, then z.r
        plain = {blocks for name, blocks, _ in launches if "k_mg_pairILi0E" in name or "k_mg_pairILi1E" in name}
        assert rc == 0 and plain, dims
        assert (nsmooth == 1) == (not named(launches, "k_mg_pairILi1E")), "plain pairs from two sweeps on"
        for blocks in plain:
            assert (blocks % columns[dims] == 0) == (dims in whole), (dims, blocks)
