"""What the host code does with errors and memory, on the CPU with the runtime's
calls faked (tests/host_cuda.py): a CUDA error that one call has returned is
not returned again by the next (the runtime keeps it until it is asked for),
a destroyed grid leaves no device memory behind, and a network has none for
a path it does not take."""
import pytest

from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
dims = (64, 80)
g, x, b = grid(dims), cells(dims), cells(dims)
result = []
for precond, refine in ((0, 0), (1, 0), (2, 0), (2, 3)):
    p, st = solver(precond=precond, refine=refine), N.PcgStats()
    solve = lambda: lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st))
    fake.fake_fail_allocation(0)
    first = solve()
    fake.fake_fail_allocation(-1)
    result.append((precond, refine, first, solve()))
    h = grid(dims)  # (the next setting allocates again)
    lib.pg_grid_destroy(g)
    g = h

# a network: its arena, then a call that checks its launches
net, params = C.c_void_p(), cells((int(lib.pg_unet_num_params()),))
fake.fake_fail_allocation(0)
first = lib.pg_unet_create(16, 16, 16, C.byref(net))
fake.fake_fail_allocation(-1)
assert lib.pg_unet_create(16, 16, 16, C.byref(net)) == 0
g = grid((16, 16, 16))
x, b = cells((16, 16, 16)), cells((16, 16, 16))
result.append(("unet", 0, first, lib.pg_unet_set_params(net, params, 1.0) or lib.pg_unet_forward_f32(net, g, b, 0.5, x)))
"""


def test_a_failed_allocation_is_reported_once(host_cuda):  # noqa: F811
    rows = host_cuda(SCRIPT)
    failed = [r for r in rows if r[2] == 7]
    assert len(failed) >= 4 and failed[-1][0] == "unet", rows
    for precond, refine, _, again in failed:
        assert again == 0, (precond, refine, again)


LEAK = r"""
result = []
for dims in ((64, 80), (32, 32, 32)):
    for precond, refine in ((0, 0), (1, 2), (2, 0), (2, 3)):
        live = fake.fake_live()
        g, x, b = grid(dims), cells(dims), cells(dims)
        p, st = solver(precond=precond, refine=refine), N.PcgStats()
        rc = lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st))
        lib.pg_grid_destroy(g)
        result.append((dims, precond, refine, rc, fake.fake_live() - live))
"""


def test_a_destroyed_grid_leaves_no_memory(host_cuda):  # noqa: F811
    for dims, precond, refine, rc, left in host_cuda(LEAK):
        assert rc == 0 and left == 0, (dims, precond, refine, rc, left)


NETWORK = r"""
V = (32, 32, 32)
g = grid(V)
solve_st, loss = N.PcgStats(), C.c_double()
empty = fake.fake_live_bytes()
net = C.c_void_p()
assert lib.pg_unet_create(*V, C.byref(net)) == 0
created = fake.fake_live_bytes()
rc, grown = [], []
for tc in ("1", "0", "0", "1"):
    os.environ["PG_UNET_TC"] = tc
    rc.append(lib.pg_unet_accumulate_f32(net, g, cells(V), cells(V), 0.5, C.byref(loss)))
    rc.append(lib.pg_solve_pressure_learned_f32(g, C.byref(solver(refine=0)), net, cells(V), cells(V), 0.5, C.byref(solve_st)))
    grown.append(fake.fake_live_bytes() - created)
lib.pg_unet_destroy(net)
lib.pg_grid_destroy(g)
result = [rc, grown, fake.fake_live_bytes()]
"""


def test_the_concatenations_are_allocated_where_they_are_written(host_cuda):  # noqa: F811
    rc, grown, left = host_cuda(NETWORK)
    assert not any(rc) and left == 0, (rc, left)
    solver_only, with_cat = grown[0], grown[1]
    cells = 32**3
    assert with_cat - solver_only == 2 * (48 * cells + 96 * cells // 8), grown
    assert grown[1:] == [with_cat] * 3
