"""z-scores bit for bit in the reference's order: vectors around the warp
width and the longest angle lists, constant and huge values, non-finite entries
(which take the ordered double sum), and in place."""
import numpy as np
import pytest
import torch

import tracetransform_gb300 as tt
from tracetransform_gb300 import autograd as tta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 359, 720, 4001])
def test_zscore_order(oracle_lib, n):
    rng = np.random.default_rng(n)
    for scale in (1e-12, 1.0, 1e9):
        x = ((rng.random(n) + rng.choice([0, 50])) * scale).astype(np.float32)
        assert np.array_equal(tt.zscore(x), oracle_lib.zscore(x))


def test_zscore_degenerate(oracle_lib):
    assert np.isnan(tt.zscore(np.float32([3.5]))).all()  # n - 1 = 0
    for c in (0.0, 0.25, 0.3):
        x = np.full(40, c, np.float32)
        assert np.array_equal(tt.zscore(x), oracle_lib.zscore(x), equal_nan=True)
    x = np.arange(70, dtype=np.float32)
    x[33] = np.inf
    assert np.isnan(tt.zscore(x)).all()
    x[33] = np.nan
    assert np.isnan(tt.zscore(x)).all()


def test_zscore_in_place():
    eng = tta.engine_for(torch.device("cuda", 0))
    x = torch.rand(500, 361, device="cuda")
    want = eng.zscore(x)
    assert torch.equal(eng.zscore(x, out=x), want)
