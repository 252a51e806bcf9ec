"""The Jacobi sweeps' rotations of V, applied beside the next sweep, at the edges of
column blocks, of chunks of block pairs and of warps' rows, against numpy."""
import numpy as np
import pytest

import tracetransform_gb300 as tt

pytestmark = pytest.mark.gpu


# one block (a bye in every round but the first), two, odd numbers of blocks, a last
# block and a last group of rows of one column, 16 and 17 pairs of blocks, columns
# past a multiple of 4 (rows of V start unaligned)
@pytest.mark.parametrize("cols", [1, 2, 11, 12, 13, 24, 25, 37, 96, 191, 383, 384, 385, 397, 601])
def test_polar_factor_over_blocks(cols):
    rng = np.random.default_rng(cols)
    rows = cols + 7
    center = (rows - 1) // 2
    sino = (0.05 * rng.random((rows, cols))).astype(np.float32)
    sino[center] += 0.05 * rows  # every column's median: no rows are added
    got, c = tt.nearest_orthonormal_sinogram(np.asfortranarray(sino))
    assert got.shape == (rows, cols) and c == center
    u, s, vt = np.linalg.svd(sino.astype(np.float64), full_matrices=False)
    # the bound of the comparison with the oracle's double Jacobi, which holds for
    # condition numbers up to 1e6
    assert s[0] / s[-1] < 1e6
    np.testing.assert_allclose(got, u @ vt, rtol=0, atol=3e-5)
