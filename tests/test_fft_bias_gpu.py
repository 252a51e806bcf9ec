"""P3 of long columns has no systematic error: over many columns the roundings of
their transforms average out, and what a root that is off in every butterfly
would leave does not."""
import numpy as np
import pytest
import torch

from tracetransform_gb300 import autograd as tta

pytestmark = pytest.mark.gpu


# rows - 1 a power of two: the functional's float linspace, and with it its weights, are
# exact.  400 columns of errors around 2.5e-7 (four times those of F) leave a mean of
# about 1e-8; allowed is one unit in the last place of the result, 2^-23.
@pytest.mark.parametrize("rows", [2049, 4097])
def test_mean_error(rows):
    eng = tta.engine_for(torch.device("cuda", 0))
    rng = np.random.default_rng(rows)
    t = np.linspace(-1, 1, rows)
    x = np.exp(-((t - rng.uniform(-0.3, 0.3, (400, 1))) / rng.uniform(0.1, 0.5, (400, 1))) ** 2)
    x = (x * rows * rng.uniform(0.1, 1, (400, 1)) + rng.uniform(0, 1, (400, rows)))
    x = x.astype(np.float32)
    got = eng.circus(torch.from_numpy(x).cuda()[None], [(3, -1, -1)])[0, 0].double().cpu().numpy()
    y = (np.abs(np.fft.fft(x.astype(np.float64), axis=1)) / rows) ** 4
    k = np.arange(rows)
    y = y[:, np.where(k <= rows // 2, k, rows - k)]
    want = (y[:, 1:] + y[:, :-1]).sum(axis=1) / (rows - 1)  # 0.5 times steps of 2 / (rows - 1)
    assert abs(np.mean(got / want - 1)) <= 2.0 ** -23
