"""The weight gradients on grids whose sides cut the 8 x 16 x 2 voxel tiles of
k_wgrad: partial rows, partial columns, an odd last plane on the coarse
levels, ranges of one tile and of several."""
import numpy as np
import pytest

from test_gpu_unet import OFFS, _case, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 36, 44), (20, 16, 28), (36, 64, 40)])
def test_weight_gradients_at_tile_edges(pg, oracle, dims):
    """Every layer within 3% relative L2 of the oracle with cosine >= 0.998:
    the bound of test_forward_and_gradients_match_oracle for the MSE loss
    (2.2% is the oracle's own sensitivity to a 1e-5 change of b)."""
    from panopaea_gb300 import learned

    g, mask, fs, b, pt, params = _case(pg, oracle, dims, seed=71 + dims[1])
    net = learned.PressureNet(dims, params=params, out_scale=3.0)
    net.set_loss(0)
    net.accumulate(g, pg.Simplex2(g, dev(b)), pg.Simplex2(g, dev(pt)), 0.5)
    grads = net.get_grads()
    _, _, ref = oracle.unet_run(params, 3.0, 0.5, dims, b, fs, pt, want_grad=True, loss_kind=0)
    for k in range(10):
        a, c = grads[OFFS[k]:OFFS[k + 1]], ref[OFFS[k]:OFFS[k + 1]]
        assert np.linalg.norm(a - c) <= 3e-2 * np.linalg.norm(c), (k, np.linalg.norm(a - c) / np.linalg.norm(c))
        assert np.vdot(a, c) >= 0.998 * np.linalg.norm(a) * np.linalg.norm(c), k
