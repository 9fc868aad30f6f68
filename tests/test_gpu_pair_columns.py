"""The fused pairs where a column of tiles gets a whole number of blocks and
where it does not: the V-cycle of separate half-sweeps, to the same bounds."""
import pytest

import test_gpu_mg as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(40, 16, 64), (9, 33, 208), (150, 72, 160), (64, 176, 320)])
def test_pairs_by_columns(pg, oracle, dims, monkeypatch):
    mg.test_fused_pairs_equal_half_sweeps(pg, oracle, dims, 1, monkeypatch)
