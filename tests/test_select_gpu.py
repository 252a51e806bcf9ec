"""The weighted selections (T6, T7, P2) where the histogram alone does not
finish them: crossing bins that hold more entries than the list, bins of equal
keys, saturated and quantised samples, the list's and the warp's edges --
every entry accounted against the oracle."""
import numpy as np
import pytest
import torch

from parity import account_circus, account_sinograms, assert_accounted, engine_sinograms
from tracetransform_gb300 import autograd as tta
from tracetransform_gb300.synthetic import blob_image

pytestmark = pytest.mark.gpu


def _image(kind):
    rng = np.random.default_rng(11)
    if kind == "narrow":  # nearly every sample in one bin of the line's range
        img = 0.5 + 1e-4 * rng.random((420, 390))
        img[200, 190] = 1.0
    elif kind == "flat":  # equal keys
        img = np.full((430, 410), 0.25)
        img[7, 9] = 1.0
    elif kind == "levels":
        img = rng.choice([0.0, 0.2, 0.8], (150, 170))
    elif kind == "saturated":
        img = np.minimum(blob_image(160, 140, 6, (20, 60), (100, 200), 3) * 1.5, 1.0)
    else:  # lines of a few samples
        img = rng.random((2, 70))
    return np.asfortranarray(img.astype(np.float32))


@pytest.mark.parametrize("kind", ["narrow", "flat", "levels", "saturated", "strip"])
def test_t6_t7(oracle_lib, kind):
    eng = tta.engine_for(torch.device("cuda", 0))
    img, tfs = _image(kind), [6, 7, 1, 3]
    ang = np.float32([0, 10, 45, 90, 133, 200, 271])
    padded = oracle_lib.pad(img)
    ref, ref_med = oracle_lib.sinograms(padded, ang, tfs, with_medians=True)
    got, got_med = engine_sinograms(eng, img, ang, tfs)
    assert_accounted(account_sinograms(padded, ang, tfs, got, ref, got_med, ref_med), kind)
    for only in ([6], [7]):  # one selection at a time: the other's does not run
        one, _ = engine_sinograms(eng, img, ang, only)
        assert np.array_equal(one[0], got[tfs.index(only[0])])


@pytest.mark.parametrize("n", [1, 31, 33, 192, 193, 260, 1449, 5793])
def test_p2(oracle_lib, n):
    eng = tta.engine_for(torch.device("cuda", 0))
    rng = np.random.default_rng(n)
    x = rng.random((n, 7))
    x[:, 1] = 3.0 + 1e-3 * x[:, 1]  # one bin, with a spike
    x[0, 1] = 40.0
    x[:, 2] = 2.5
    x[:, 3] = rng.choice([0.0, 1.0, 5.0], n)
    x[:, 4] = 0.0
    x[:, 5] = 1e-30 * x[:, 5]
    x[:, 6] = np.where(rng.random(n) < 0.02, 1e4, x[:, 6] * 1e-3)
    x = np.asfortranarray(x.astype(np.float32))
    got = eng.circus(torch.from_numpy(np.ascontiguousarray(x.T)).cuda()[None], [(2, -1, -1)])
    assert_accounted(account_circus(x[None], [(2, 0, 0)], got.cpu().numpy()), str(n))
