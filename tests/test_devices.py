"""What the host code finds out about a kernel (its shared-memory opt-in, the
blocks that fit an SM) holds for one device, and a failure to find it out is
not kept.  With the runtime faked: a launch with more shared memory than the
kernel was opted into on the current device fails, as it does in CUDA."""
from host_cuda import host_cuda  # noqa: F401

SCRIPT = r"""
V, H, B2 = (32, 32, 32), (300, 281), (40, 70)
x, b, vel, rho = (cells((200000,)) for _ in range(4))
params = cells((int(lib.pg_unet_num_params()),))
hs, ws = (C.c_int64 * 2)(300, 60), (C.c_int64 * 2)(300, 70)

def work(device):
    '''Solves, a step and a network on a device: the statuses and the kernels.'''
    fake.fake_set_device(device)
    rc, st, loss = [], N.PcgStats(), C.c_double()
    log()
    for dims in (V, H, B2):
        g = grid(dims)
        for precond, refine in ((0, 0), (1, 0), (2, 0), (2, 2)):
            p = solver(precond=precond, refine=refine)
            rc.append(lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st)))
        lib.pg_grid_destroy(g)
    os.environ["PG_MG_CTAIL"] = "0"
    g = grid(V)
    p = solver(precond=2)
    rc.append(lib.pg_solve_pressure_f32(g, C.byref(p), x, b, 0.5, C.byref(st)))
    del os.environ["PG_MG_CTAIL"]
    rc.append(lib.pg_pcg_f64(g, 0, cells(V, 8), cells(V, 8), 5, 1e-9, cells(V, 8), cells(V, 8), cells(V, 8), 0.5, C.byref(st)))
    B = C.c_void_p()
    rc.append(lib.pg_batch_create_2d(2, hs, ws, C.byref(B)))
    sp = N.StepParams()
    sp.dt, sp.solver = 0.5, solver(precond=2)
    rc.append(lib.pg_batch_step_f32(B, C.byref(sp), cells((400000,)), rho, x, (N.PcgStats * 2)()))
    lib.pg_batch_destroy(B)
    net = C.c_void_p()
    rc.append(lib.pg_unet_create(*V, C.byref(net)) or lib.pg_unet_set_params(net, params, 1.0))
    for tc in ("1", "0"):
        os.environ["PG_UNET_TC"] = tc
        rc.append(lib.pg_unet_forward_f32(net, g, b, 0.5, x))
        rc.append(lib.pg_unet_accumulate_f32(net, g, b, x, 0.5, C.byref(loss)))
    lib.pg_unet_destroy(net)
    lib.pg_grid_destroy(g)
    return rc, kernels()
"""

TWO = SCRIPT + r"""
a, b_ = work(0), work(1)
result = [a[0], b_[0], a[1] == b_[1], lib.pg_last_error().decode()]
"""


def test_a_second_device(host_cuda):  # noqa: F811
    first, second, same, message = host_cuda(TWO)
    assert not any(first), (first, message)
    assert not any(second) and same, (second, message)


FAILURES = SCRIPT + r"""
want = work(0)
result = []
for k in range(60):
    fake.fake_fail_attribute(k)
    work(1 + k)  # (it may fail, or take another way)
    fake.fake_fail_attribute(-1)
    got = work(1 + k)
    result.append((k, got[0], got[1] == want[1]))
"""


def test_a_failed_query_is_not_kept(host_cuda):  # noqa: F811
    for k, rc, same in host_cuda(FAILURES):
        assert not any(rc) and same, (k, rc)


HEAD = r"""
V = (48, 48, 48)
result = []
for sms in (152, 100):
    fake.fake_set_sms(sms)
    g, net, loss = grid(V), C.c_void_p(), C.c_double()
    assert lib.pg_unet_create(*V, C.byref(net)) == 0
    log()
    rc = lib.pg_unet_accumulate_f32(net, g, cells(V), cells(V), 0.5, C.byref(loss))
    result.append((sms, rc, [n for k, n, _ in log() if "6k_head" in k]))
"""


def test_the_loss_runs_on_every_sm(host_cuda):  # noqa: F811
    """The last launch, the one with the FP64 sums, has as many blocks for every SM."""
    for sms, rc, blocks in host_cuda(HEAD):
        assert rc == 0 and blocks[-1] == min(4 * sms, 48**3 // 256), (sms, blocks)
