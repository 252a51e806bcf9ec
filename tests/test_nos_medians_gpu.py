"""The weighted medians that align a sinogram's columns, against numpy."""
import numpy as np
import pytest

import tracetransform_gb300 as tt
from tracetransform_gb300._native import TTError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 15, 16, 17, 31, 33, 47, 260])
def test_alignment_medians(rows):
    """The aligned rows and the center follow from every column's weighted
    median of sequential float sums; zero, negative and tying columns among them."""
    rng = np.random.default_rng(rows)
    cols = min(rows, 9)
    sino = rng.random((rows, cols)).astype(np.float32)
    if cols > 3:
        sino[:, 1] = 0
        sino[:, 2] = 1  # 2 * prefix == total at the middle
        sino[:, 3] -= 0.7
    prefix = np.cumsum(sino, axis=0, dtype=np.float32)
    hit = 2 * prefix >= prefix[-1]
    median = np.where(hit.any(0), hit.argmax(0), rows - 1)
    center = (rows - 1) // 2
    mx, mn = int((median - center).max()), int((median - center).min())
    got, c = tt.nearest_orthonormal_sinogram(np.asfortranarray(sino))
    assert got.shape == (rows + abs(mx) + abs(mn), cols)
    assert c == center + mx


@pytest.mark.parametrize("rows", [8190, 8191, 8193, 9001])
def test_longest_columns(rows):
    """Up to 8192 aligned rows are taken; more are refused with their number,
    whichever kernel finds the medians."""
    rng = np.random.default_rng(rows)
    sino = (0.05 * rng.random((rows, 3))).astype(np.float32)
    sino[(rows - 1) // 2 + 1] += rows  # every median one row past the center: |1| + |1| rows more
    if rows + 2 <= 8192:
        got, c = tt.nearest_orthonormal_sinogram(np.asfortranarray(sino))
        assert got.shape == (rows + 2, 3) and c == (rows - 1) // 2 + 1
    else:
        with pytest.raises(TTError, match=f"{rows + 2} aligned rows exceeds 8192"):
            tt.nearest_orthonormal_sinogram(np.asfortranarray(sino))
