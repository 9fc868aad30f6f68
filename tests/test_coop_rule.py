"""Which double grids the cooperative CG takes (host code, runtime faked): none
whose rows or planes are so large beside a block's cells that the loop of two
kernels is faster, and threads for the halo on the ones it takes."""
import pytest

from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
result = []
for dims in %r:
    n = 1
    for d in dims:
        n *= d
    for precond in (0, 1):
        g = grid(dims)
        v = [cells(dims, 8) for _ in range(5)]
        st = N.PcgStats()
        log()
        rc = lib.pg_pcg_f64(g, precond, v[0], v[1], 10, 1e-9, v[2], v[3], v[4], 0.5, C.byref(st))
        coop = [(b, t) for k, b, t in log() if "k_cg_coop" in k]
        result.append((dims, precond, rc, coop))
        lib.pg_grid_destroy(g)
        keep.clear()
"""

TAKEN = [(1, 3), (16, 16), (128, 128), (384, 384), (33, 901), (10, 3000), (30, 4000), (25, 10000), (700, 800),
         (3, 20, 20), (9, 20, 31), (64, 64, 64), (4, 64, 64), (16, 80, 80), (12, 100, 100), (60, 100, 100), (64, 64, 150)]
# (900 x 900: too many cells; 40 x 109 x 109: the planes do not fit shared memory)
LEFT = [(2, 8000), (5, 5000), (10, 8000), (8, 12000), (18, 9000), (900, 900), (2, 85, 85), (8, 100, 100), (12, 90, 90),
        (10, 95, 95), (40, 109, 109)]


@pytest.mark.parametrize("taken", [True, False])
def test_route(host_cuda, taken):  # noqa: F811
    for dims, precond, rc, coop in host_cuda(SCRIPT % (TAKEN if taken else LEFT)):
        assert rc == 0 and len(coop) == (1 if taken else 0), (dims, precond, rc, coop)
        if taken:
            blocks, threads = coop[0]
            halo = 2 * (dims[-1] if len(dims) == 2 else dims[-1] * dims[-2])
            assert threads == 512 or 8 * threads >= halo, (dims, blocks, threads)
