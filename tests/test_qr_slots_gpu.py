"""The pivoted QR at the edges of its row slots and column groups, against numpy."""
import numpy as np
import pytest

import tracetransform_gb300 as tt

pytestmark = pytest.mark.gpu


# aligned rows around one slot of a CTA (128, 256, 512 rows) and the classes' limits;
# angles that leave a part of a group, one column, and more columns than rows of a slot
@pytest.mark.parametrize("rows,cols", [(33, 33), (127, 5), (128, 1), (129, 129), (255, 18),
                                       (257, 200), (511, 41), (512, 40), (513, 41), (1023, 7),
                                       (1025, 33), (1280, 9), (1281, 34), (2047, 12), (2049, 13),
                                       (4096, 6)])
def test_polar_factor_at_slot_edges(rows, cols):
    rng = np.random.default_rng(rows * 1000 + cols)
    center = (rows - 1) // 2
    sino = (0.05 * rng.random((rows, cols))).astype(np.float32)
    sino[center] += 0.05 * rows  # every column's median: no rows are added
    got, c = tt.nearest_orthonormal_sinogram(np.asfortranarray(sino))
    assert got.shape == (rows, cols) and c == center
    u, _, vt = np.linalg.svd(sino.astype(np.float64), full_matrices=False)
    # the bound of the comparison with the oracle's double Jacobi
    np.testing.assert_allclose(got, u @ vt, rtol=0, atol=2e-5)
