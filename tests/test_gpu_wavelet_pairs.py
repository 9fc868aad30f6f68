"""The wavelet passes with four pairs per thread, halves that are no multiple
of four and blocks that several rows share: bit for bit against the oracle,
special values included.  (Which sizes take four: tests/test_wavelet_pairs.py.)"""
import numpy as np
import pytest

from conftest import rng
from test_gpu_wavelet_pass import both_ways

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("wavelet", range(5))
def test_four_pairs_bit_exact(pg, oracle, wavelet, special):
    shape = (470, 490) if wavelet in (2, 3) else (1524, 756)
    r = rng(wavelet + 100 * special)
    X = r.standard_normal(shape)
    if special:
        X[r.random(shape) < 0.3] = 0.0
        X[r.random(shape) < 0.2] = -0.0
        X[3, 5], X[-2, 1], X[17, -1], X[20, 20], X[-1, 300] = np.inf, -np.inf, np.nan, 1e308, np.inf
    both_ways(oracle, X, wavelet, wavelet, 1)
