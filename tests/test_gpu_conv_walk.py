"""The walking tensor-core convolutions: several tiles per CTA (so that stages,
accumulator sets and barrier phases come round), both tile depths, grids
whose last tiles are cut in every direction, and the concatenations read
where they are (forward) or written out (training)."""
import numpy as np
import pytest

from test_gpu_unet import _case, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(100, 72, 84), (16, 144, 132), (84, 20, 200), (16, 16, 20)])
def test_forward_and_loss_match_warp_mma(pg, oracle, dims, monkeypatch):
    """Against the mma.sync kernel, whose FP32 sums run in another order: a
    BF16 activation flips by 2^-8 now and then, ten layers deep: 1% of the
    output's norm, 1e-3 of the loss."""
    from panopaea_gb300 import _native as N
    from panopaea_gb300 import learned

    g, mask, fs, b, pt, params = _case(pg, oracle, dims, seed=7 + dims[2])
    gb, gpt = pg.Simplex2(g, dev(b)), pg.Simplex2(g, dev(pt))
    res = {}
    for tc in ("1", "0"):
        monkeypatch.setenv("PG_UNET_TC", tc)
        net = learned.PressureNet(dims, params=params, out_scale=3.0)
        x = g.new_simplex_2()
        net.forward(g, gb, 0.5, x)
        first = host(x)
        net.forward(g, gb, 0.5, x)
        assert np.array_equal(first, host(x))
        loss = net.accumulate(g, gb, gpt, 0.5)
        assert N.load().pg_unet_check(net._h) == N.PG_OK
        res[tc] = (first, loss)
    (x1, l1), (x0, l0) = res["1"], res["0"]
    assert np.linalg.norm(x1 - x0) <= 1e-2 * np.linalg.norm(x0)
    assert abs(l1 - l0) <= 1e-3 * l0
