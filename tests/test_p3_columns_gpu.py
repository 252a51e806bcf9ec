"""P3 of a column is its own whatever the columns beside it: few and many columns, whole and
partial tiles of 128, and columns of fewer, as many and more stages of 32 rows than
the tensor-core DFT's ring holds."""
import numpy as np
import pytest
import torch

from tracetransform_gb300 import autograd as tta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 31, 32, 33, 64, 65, 96, 97, 128, 129, 363, 1449, 2048])
def test_p3_of_a_column_is_its_own(rows):
    eng = tta.engine_for(torch.device("cuda", 0))
    rng = np.random.default_rng(rows)
    x = torch.from_numpy((rng.random((1, 400, rows)) * 50).astype(np.float32)).cuda()
    pf = [(3, -1, -1)]
    whole = eng.circus(x, pf)[0, 0]
    for first, count in ((0, 1), (5, 15), (0, 16), (3, 17), (11, 45), (0, 64), (100, 127),
                         (100, 128), (7, 129), (0, 257)):
        part = eng.circus(x[:, first:first + count].contiguous(), pf)[0, 0]
        assert torch.equal(part, whole[first:first + count])
    # many tiles in flight, the same again
    big = x.repeat(12, 1, 1)
    assert torch.equal(eng.circus(big, pf)[:, 0], whole.expand(12, -1))
    y = (np.abs(np.fft.fft(x[0].cpu().numpy().astype(np.float64), axis=1)) / rows) ** 4
    k = np.arange(rows)
    y = y[:, np.where(k <= rows // 2, k, rows - k)]
    lin = (-1 + k * 2.0 / (rows - 1)).astype(np.float32).astype(np.float64)
    want = (0.5 * np.diff(lin) * (y[:, 1:] + y[:, :-1])).sum(axis=1)
    # FP32 accumulation of rows / 8 matrix products, fourth power: 4 * 2^-24 * rows / 24 and the
    # split's 4 * 2^-21, on a mean that carries at least half the norm
    tol = 2 * (4 * 2.0 ** -24 * max(rows / 24, 4) + 4 * 2.0 ** -21)
    np.testing.assert_allclose(whole.double().cpu().numpy(), want, rtol=tol)
