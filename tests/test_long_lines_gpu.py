"""Lines long enough for four warps each (more than 8 lines' buffers in half an
SM's shared memory): every split of the T-functionals over them, and the
longest lines the engine takes."""
import numpy as np
import pytest
import torch

from parity import account_sinograms, assert_accounted, engine_sinograms
from tracetransform_gb300 import autograd as tta
from tracetransform_gb300._native import TTError
from tracetransform_gb300.api import pad_geometry
from tracetransform_gb300.synthetic import blob_image

pytestmark = pytest.mark.gpu
ANG = np.float32([0, 17, 90])


@pytest.fixture(scope="module")
def strip(oracle_lib):
    """A 4100 x 50 image, its frame and the oracle's sinograms."""
    img = blob_image(4100, 50, 12, (10, 300), (40, 200), 31)
    padded = oracle_lib.pad(img)
    ref, med = oracle_lib.sinograms(padded, ANG, list(range(8)), with_medians=True)
    return img, padded, ref, med


@pytest.mark.parametrize("tfs", [[0], [1, 2], [2, 0], [3], [5, 4, 3], [6], [7], [7, 6], [0, 6],
                                 [1, 4, 7], [0, 1, 2, 3, 4, 5], list(range(8)),
                                 [6, 6, 7, 0, 1, 2, 3, 4, 5, 7]])
def test_functional_sets(strip, tfs):
    eng = tta.engine_for(torch.device("cuda", 0))
    img, padded, ref, med = strip
    got, got_med = engine_sinograms(eng, img, ANG, tfs)
    rep = account_sinograms(padded, ANG, tfs, got, ref[tfs], got_med, med[tfs])
    assert_accounted(rep, str(tfs))


@pytest.mark.parametrize("tfs,n", [([0, 6], 13727), ([0, 5], 14495)])
def test_longest_lines(tfs, n):
    """The longest line whose buffers fit shared memory still runs; the next
    one is refused."""
    eng = tta.engine_for(torch.device("cuda", 0))
    rows = next(r for r in range(n - 8, n) if pad_geometry(r, 3)[0] == n)
    img = torch.rand(3, rows, device="cuda")
    out = eng.sinograms(img, rows, 3, [0.0], tfs)
    assert torch.isfinite(out).all()
    # angle 0: the columns' sums, of the rows the reference samples (0 <= q < n - 1)
    seen = img[:, :n - 1 - pad_geometry(rows, 3)[1]]
    assert out[0, 0].double().sum().item() == pytest.approx(seen.double().sum().item(), rel=1e-5)
    assert float(out[1].abs().max()) > 0
    rows = next(r for r in range(n, n + 80) if pad_geometry(r, 3)[0] > n + 64)
    with pytest.raises(TTError):
        eng.sinograms(torch.rand(3, rows, device="cuda"), rows, 3, [0.0], tfs)
