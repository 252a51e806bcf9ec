"""T6 and T7 of lines with hardly any light: over a range below 2^-120 the
reciprocal of a histogram bin's width is no float, yet a line's zeros and
samples must not share one bin.  (Normal floats only: the texture reads
subnormal pixels as zeros.)"""
import numpy as np
import pytest
import torch

from parity import engine_sinograms
from tracetransform_gb300 import autograd as tta

pytestmark = pytest.mark.gpu


def _sparse(rows):
    """Columns of zeros, one bright pixel on the median's side and 60 others after
    it, in multiples of 1/16: sums and products with rows exact in float."""
    rng = np.random.default_rng(rows)
    img = np.zeros((rows, 12), np.float32)
    for c in range(12):
        at = np.sort(rng.choice(np.arange(rows // 8, rows - 4), 60, replace=False))
        img[at, c] = rng.integers(16, 64, 60) / 16
        img[rows // 8 - 1, c] = 34
    return np.asfortranarray(img)


# Unrotated lines are the image's columns, a power of four scales every sample,
# sum, root and key exactly, and the selections scale with them.
@pytest.mark.parametrize("rows", [150, 260, 600, 2900])
@pytest.mark.parametrize("e", [60, 112, 116, 120, 122, 124, 126])
def test_t6_t7_scale_exactly(rows, e):
    eng = tta.engine_for(torch.device("cuda", 0))
    img, ang = _sparse(rows), np.float32([0])
    want, want_med = engine_sinograms(eng, img, ang, [6, 7])
    got, med = engine_sinograms(eng, np.asfortranarray(img * np.float32(2.0 ** -e)), ang, [6, 7])
    assert ((want[:, :, 0] > 0).sum(axis=1) == 12).all()
    assert np.array_equal(med, want_med)
    assert np.array_equal(got, (want.astype(np.float64) * 2.0 ** -e).astype(np.float32))


@pytest.mark.parametrize("e", [0, 60, 96, 100, 110, 120])
def test_t6_t7_neighbouring_floats(e):
    """More samples than the list holds, of three neighbouring floats each: the
    crossing bin is refined down to single keys."""
    eng = tta.engine_for(torch.device("cuda", 0))
    rng = np.random.default_rng(3)
    ulp = np.float32(2.0 ** -23)
    img = np.asfortranarray((1 + ulp * rng.integers(0, 3, (700, 9))).astype(np.float32))
    img[20] = 40
    ang = np.float32([0])
    want, want_med = engine_sinograms(eng, img, ang, [6, 7])
    got, med = engine_sinograms(eng, np.asfortranarray(img * np.float32(2.0 ** -e)), ang, [6, 7])
    assert np.array_equal(med, want_med)
    assert np.array_equal(got, (want.astype(np.float64) * 2.0 ** -e).astype(np.float32))
