"""A multigrid hierarchy whose build fails part way (no memory for one of its
arrays) is not kept: the next solve on the same mask and time step builds it
again, from the first allocation to the last setup kernel.  On the CPU, with
the runtime's calls faked (tests/host_cuda.py)."""
import pytest

from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
dims = %(dims)r
p = solver(precond=2, refine=0)
x, b = cells(dims), cells(dims)
st = N.PcgStats()

def solve(g):
    rc = lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st))
    return rc, kernels()

setup = ("k_mg_coarsen", "k_mg_invd", "k_mg_pack")
def built(names):
    return [n for n in names if any(s in n for s in setup)]

# an undisturbed first solve: its allocations and setup kernels
g = grid(dims)
log()
n0 = fake.fake_allocations()
rc, names = solve(g)
assert rc == 0, (rc, lib.pg_last_error())
want, allocations = built(names), fake.fake_allocations() - n0
assert want and allocations > 3, (want, allocations)
rc, names = solve(g)  # kept: nothing is built again
assert rc == 0 and not built(names)
lib.pg_grid_destroy(g)
live = fake.fake_live()

result = []
for k in range(allocations):
    g = grid(dims)
    log()
    fake.fake_fail_allocation(k)
    rc, names = solve(g)
    fake.fake_fail_allocation(-1)
    second, again = solve(g)
    # (what the first call built before it failed elsewhere is kept)
    whole = built(again) == want or (built(names) == want and not built(again))
    lib.pg_grid_destroy(g)
    result.append((k, rc, second, whole, fake.fake_live() - live))
"""


@pytest.mark.parametrize("dims", [(97, 131), (700, 130), (30, 33, 35), (32, 32, 32)])
def test_failed_build_is_not_kept(host_cuda, dims):  # noqa: F811
    rows = host_cuda(SCRIPT % dict(dims=dims))
    assert len(rows) > 3
    for k, first, second, whole, leaked in rows:
        assert first == 7, ("the failed allocation is reported", k, first)
        assert second == 0, ("the next solve succeeds", k, second)
        assert whole, ("and build the whole hierarchy", k)
        assert leaked == 0, (k, leaked)
