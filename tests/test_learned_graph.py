"""The captured CG loop of a learned solve is replayed only for the kernel
sequence it was captured from (host code, runtime faked)."""
from host_cuda import host_cuda  # noqa: F401

PRE = r"""
dims = (16, 16, 16)
g, x, b = grid(dims), cells(dims), cells(dims)
params = cells((int(lib.pg_unet_num_params()),))

def network():
    net = C.c_void_p()
    assert lib.pg_unet_create(*dims, C.byref(net)) == 0
    assert lib.pg_unet_set_params(net, params, 1.0) == 0
    return net

def solve(net):
    st = N.PcgStats()
    p = solver(refine=0)
    log()
    rc = lib.pg_solve_pressure_learned_f32(g, C.byref(p), net, x, b, 0.5, C.byref(st))
    names = kernels()
    return rc, [sum(k in n for n in names) for k in ("k_conv_tc", "6k_convI")]
"""

SWITCH = PRE + r"""
net = network()
result = []
for tc in ("1", "0", "1", "0"):
    os.environ["PG_UNET_TC"] = tc
    result.append((tc,) + solve(net))
"""


def test_the_convolution_switch_is_part_of_the_key(host_cuda):  # noqa: F811
    """A loop captured with the tensor-core convolutions reads their weight
    layout; the other setting brings only its own up to date."""
    for tc, rc, (tensor, warp) in host_cuda(SWITCH):
        assert rc == 0
        # ten layers for the first application and ten in the loop
        assert (tensor, warp) == ((20, 0) if tc == "1" else (0, 20)), (tc, tensor, warp)


REPLACED = PRE + r"""
result = []
for _ in range(8):
    net = network()
    first = net.value
    before = fake.fake_captures()
    solve(net), solve(net)
    result.append((first, fake.fake_captures() - before))
    lib.pg_unet_destroy(net)
"""


def test_a_network_at_the_address_of_another_gets_its_own_loop(host_cuda):  # noqa: F811
    """The loop holds the network's buffers; those of a destroyed one are freed."""
    rows = host_cuda(REPLACED)
    assert len({at for at, _ in rows}) < len(rows)  # an address came back
    assert [n for _, n in rows] == [1] * len(rows), rows
