"""The chirp-z transforms of column pairs: P3 of columns over 2048 rows and the
P-stage adjoint against float64, at the transform lengths' edges, with odd
column counts, and with columns that must not disturb their neighbour (zero,
tiny, non-finite)."""
import numpy as np
import pytest
import torch

from tracetransform_gb300 import autograd as tta

pytestmark = pytest.mark.gpu


def _columns(rows, cols, seed):
    """Positive bumps with noise: (1, cols, rows) float32 on the device."""
    rng = np.random.default_rng(seed)
    t = np.linspace(-1, 1, rows)
    x = np.exp(-((t - rng.uniform(-0.3, 0.3, (cols, 1))) / rng.uniform(0.1, 0.5, (cols, 1))) ** 2)
    x = x * rows * rng.uniform(0.1, 1, (cols, 1)) + rng.uniform(0, 1, (cols, rows))
    return torch.from_numpy(x.astype(np.float32)).cuda()[None]


def _p3(x):
    """P3 in float64 with the linspace rounded to float32, as the functional
    defines it (x: (cols, rows))."""
    n = x.shape[1]
    y = (np.abs(np.fft.fft(x.astype(np.float64), axis=1)) / n) ** 4
    k = np.arange(n)
    y = y[:, np.where(k <= n // 2, k, n - k)]
    lin = (-1 + k * 2.0 / (n - 1)).astype(np.float32).astype(np.float64)
    return (0.5 * np.diff(lin) * (y[:, 1:] + y[:, :-1])).sum(axis=1)


# float FFT: about log2(M) roundings of 2^-24 each way on a signal whose mean
# carries at least half its norm, four times that in |F|^4: 4 * 2 * 28 * 2^-24
P3_TOL = 1.4e-5


@pytest.mark.parametrize("rows,cols", [(2049, 2), (4096, 3), (4097, 1), (5793, 7), (8192, 2)])
def test_p3_long_columns(rows, cols):
    eng = tta.engine_for(torch.device("cuda", 0))
    x = _columns(rows, cols, rows)
    got = eng.circus(x, [(3, -1, -1)])[0, 0].double().cpu().numpy()
    np.testing.assert_allclose(got, _p3(x[0].cpu().numpy()), rtol=P3_TOL)


def test_p3_long_columns_keep_their_neighbours_out():
    eng = tta.engine_for(torch.device("cuda", 0))
    x = _columns(3001, 10, 5)
    x[0, 1] *= 1e-9
    x[0, 3] = 0
    x[0, 4, 17] = float("inf")
    x[0, 7, 100] = float("nan")
    x[0, 8] *= 1e15  # the square of its norm overflows at x[9]'s scale
    got = eng.circus(x, [(3, -1, -1)])[0, 0].double().cpu().numpy()
    want = _p3(x[0].cpu().numpy())
    assert got[3] == 0 and not np.isfinite(got[4]) and np.isnan(got[7])
    for c in (0, 2, 5, 6, 9):
        np.testing.assert_allclose(got[c], want[c], rtol=P3_TOL)
    tiny = eng.circus(x[:, 1:2].contiguous(), [(3, -1, -1)])[0, 0, 0].item()
    assert got[1] == pytest.approx(tiny, rel=2 * P3_TOL, abs=1e-44)


@pytest.mark.parametrize("rows,cols", [(17, 2), (32, 3), (33, 2), (64, 2), (65, 1), (128, 5),
                                       (129, 2), (363, 3), (512, 2), (513, 2), (1024, 2),
                                       (2048, 3), (4097, 2), (8192, 2)])
def test_adjoint_pairs(rows, cols):
    """Float against float64 adjoint: each column within 1e-4 of its largest
    entry (the transforms' 1e-5 and the float sums of the float64 comparison)."""
    eng = tta.engine_for(torch.device("cuda", 0))
    x = _columns(rows, cols, rows + 1)
    pf = [(1, -1, -1), (3, -1, -1)]
    g = torch.from_numpy(np.random.default_rng(rows).standard_normal((1, 2, cols))).cuda()
    g[0, 0] = 0  # P3 alone: P1's signs would hide it
    got = eng.circus_backward(x, pf, g.float().contiguous()).double()
    want = eng.circus_backward(x.double(), pf, g)
    err = (got - want).abs().amax(-1) / want.abs().amax(-1)
    assert float(err.max()) <= 1e-4, err


def test_adjoint_pairs_keep_their_neighbours_out():
    eng = tta.engine_for(torch.device("cuda", 0))
    x = _columns(363, 8, 9)
    x[0, 1] *= 1e-6
    x[0, 3] = 0
    x[0, 4, 17] = float("nan")
    x[0, 7] *= 1e18  # |F|^2 F overflows
    pf = [(3, -1, -1)]
    g = torch.ones((1, 1, 8), device="cuda")
    g[0, 0, 6] = 0
    got = eng.circus_backward(x, pf, g)
    assert torch.all(got[0, 3] == 0) and torch.all(got[0, 6] == 0)
    assert torch.isnan(got[0, 4]).all()
    for c in (0, 1, 2, 5):
        one = eng.circus_backward(x[:, c:c + 1].contiguous(), pf, g[:, :, c:c + 1].contiguous())
        scale = one.abs().max()
        assert float((got[0, c] - one[0, 0]).abs().max()) <= 1e-4 * float(scale)
