"""The wavelet pass kernels at the sizes where they can go wrong -- lines just
above twice the filter length, halves that are no multiple of a thread's four
pairs, rows of several segments -- and on infinities, NaN and signed zeros:
bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import rng

pytestmark = pytest.mark.gpu

TAPS = (2, 6, 6, 10, 4)


def same_bits(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a[~nan].view(np.int64), b[~nan].view(np.int64))


def both_ways(oracle, X, wx, wy, levels):
    import torch

    from panopaea_gb300 import wavelet as WV

    for fmode, imode in ((0, 0), (1, 2)):
        t = torch.from_numpy(X.copy()).cuda()
        WV.fwt_2d(t, levels, wx, wy, mode=fmode)
        Y = oracle.wavelet_fwt_2d(fmode, wx, wy, X, levels)
        assert same_bits(t.cpu().numpy(), Y), fmode
        WV.ifwt_2d(t, levels, wx, wy, mode=imode)
        assert same_bits(t.cpu().numpy(), oracle.wavelet_ifwt_2d(imode, wx, wy, Y, levels)), imode


@pytest.mark.parametrize("wx,wy", [(0, 3), (1, 4), (2, 2), (3, 0), (4, 1)])
@pytest.mark.parametrize("shape,levels", [((20, 22), 1), ((62, 38), 1), ((516, 604), 2), ((290, 1030), 1)])
def test_passes_bit_exact(pg, oracle, wx, wy, shape, levels):
    if (shape[1] >> (levels - 1)) < TAPS[wx] or (shape[0] >> (levels - 1)) < TAPS[wy]:
        pytest.skip("last level shorter than the filter")
    both_ways(oracle, rng(shape[0] + 5 * wx + wy).standard_normal(shape), wx, wy, levels)


@pytest.mark.parametrize("wavelet", range(5))
@pytest.mark.parametrize("shape", [(48, 40), (400, 512)])
def test_special_values(pg, oracle, wavelet, shape):
    r = rng(wavelet + shape[0])
    X = r.standard_normal(shape)
    X[r.random(shape) < 0.3] = 0.0
    X[r.random(shape) < 0.2] = -0.0
    X[3, 5], X[-2, 1], X[17, -1], X[20, 20] = np.inf, -np.inf, np.nan, 1e308
    X[30:34, 8:30] = -0.0
    both_ways(oracle, X, wavelet, wavelet, 1)


def test_lines_of_one_dimension(pg, oracle):
    import torch

    from panopaea_gb300 import wavelet as WV

    for wavelet in range(5):
        for n, levels in ((20, 1), (1 << 16, 6), (3 * 4096, 5)):
            x = rng(n + wavelet).standard_normal(n)
            t = torch.from_numpy(x.copy()).cuda()
            WV.fwt_1d(t, levels, wavelet)
            y = oracle.wavelet_fwt_1d(wavelet, x, levels)
            assert same_bits(t.cpu().numpy(), y)
            WV.ifwt_1d(t, levels, wavelet)
            assert same_bits(t.cpu().numpy(), oracle.wavelet_ifwt_1d(wavelet, y, levels))
