"""Square-root weights (T3-T7) of lines with samples outside the branch-free
root's range -- tiny, negative and subnormal pixels -- beside ordinary ones."""
import numpy as np
import pytest
import torch

from parity import account_sinograms, assert_accounted, engine_sinograms
from tracetransform_gb300 import autograd as tta
from tracetransform_gb300.synthetic import blob_image

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tfs", [[3, 4, 5], [0, 1, 2, 3, 4, 5, 6, 7]])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -80, 2.0 ** -110])
def test_small_samples(oracle_lib, tfs, scale):
    """Scaled images, the darkest pixels of a mixed one scaled further: the
    samples cross the range's lower end inside a line."""
    eng = tta.engine_for(torch.device("cuda", 0))
    img = blob_image(60, 47, 5, (4, 12), (40, 200), 21).astype(np.float64) * scale
    img[20:30] *= 2.0 ** -40
    img = np.asfortranarray(img.astype(np.float32))
    ang = np.float32([0, 13, 90, 200])
    padded = oracle_lib.pad(img)
    ref, ref_med = oracle_lib.sinograms(padded, ang, tfs, with_medians=True)
    got, got_med = engine_sinograms(eng, img, ang, tfs)
    assert_accounted(account_sinograms(padded, ang, tfs, got, ref, got_med, ref_med), str(scale))


def test_negative_pixels_reach_the_general_root(oracle_lib):
    """A negative pixel makes the lines that sample it NaN in the root sums
    and leaves every other line as it is without the pixel."""
    eng = tta.engine_for(torch.device("cuda", 0))
    img = blob_image(40, 40, 4, (4, 12), (40, 200), 5)
    bad = img.copy(order="F")
    bad[11, 17] = -0.5
    ang = np.float32([0, 90])
    a, _ = engine_sinograms(eng, img, ang, [0, 3, 5])
    b, _ = engine_sinograms(eng, bad, ang, [0, 3, 5])
    same = np.isclose(a[0], b[0], rtol=1e-6)
    assert np.array_equal(a[1:, same], b[1:, same])
    assert 0 < (~same).sum() <= 6
