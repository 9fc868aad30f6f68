"""A kernel that cannot be launched -- also while a solver loop is captured,
where the loop would run without it, without its end if it is the one that
ends it -- fails the call, and the next call captures the whole loop.  Host
code, runtime faked."""
import pytest

from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
which = %r
V = (32, 32, 32)
x, b, vel, rho = (cells((200000,)) for _ in range(4))
st = N.PcgStats()

def solver_case(dims, **kw):
    def solve(g):
        return lib.pg_solve_pressure_f32(g, C.byref(solver(**kw)), x, b, 0.5, C.byref(st))
    return lambda: grid(dims), solve, lib.pg_grid_destroy

def batch_case(precond):
    def make():
        B = C.c_void_p()
        assert lib.pg_batch_create_2d(2, (C.c_int64 * 2)(300, 60), (C.c_int64 * 2)(300, 70), C.byref(B)) == 0
        return B
    def step(B):
        sp = N.StepParams()
        sp.dt, sp.solver = 0.5, solver(precond=precond)
        return lib.pg_batch_step_f32(B, C.byref(sp), vel, rho, x, (N.PcgStats * 2)())
    return make, step, lib.pg_batch_destroy

def learned_case():
    g = grid(V)
    params = cells((int(lib.pg_unet_num_params()),))
    def make():
        net = C.c_void_p()
        assert lib.pg_unet_create(*V, C.byref(net)) == 0 and lib.pg_unet_set_params(net, params, 1.0) == 0
        return net
    def solve(net):
        return lib.pg_solve_pressure_learned_f32(g, C.byref(solver(refine=0)), net, x, b, 0.5, C.byref(st))
    return make, solve, lib.pg_unet_destroy

make, call, free = {
    "cg": lambda: solver_case((60, 70), precond=0), "jacobi": lambda: solver_case(V, precond=1),
    "mg2d": lambda: solver_case((300, 281), precond=2, refine=2), "mg3d": lambda: solver_case(V, precond=2, refine=2),
    "batch": lambda: batch_case(0), "batch_mg": lambda: batch_case(2), "learned": learned_case,
}[which]()

o = make()
log()
assert call(o) == 0
first = len(log())
assert call(o) == 0
want = kernels()
free(o)
result = []
for k in range(first):
    o = make()
    fake.fake_fail_launch(k)
    failed = call(o)
    fake.fake_fail_launch(-1)
    again = call(o)
    log()
    third = call(o)
    result.append((k, failed, again, third, kernels() == want))
    free(o)
"""


@pytest.mark.parametrize("which", ["cg", "jacobi", "mg2d", "mg3d", "batch", "batch_mg", "learned"])
def test_a_failed_launch_fails_the_call(host_cuda, which):  # noqa: F811
    rows = host_cuda(SCRIPT % which)
    assert len(rows) >= 4
    for k, failed, again, third, whole in rows:
        assert failed in (5, 7), ("the launch that failed is reported", k, failed)
        assert again == 0 and third == 0 and whole, ("and the loop is whole afterwards", k, again, third, whole)
