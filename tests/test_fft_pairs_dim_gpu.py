"""Dim columns in the chirp-z transforms of column pairs: a column whose squared
norm (its own, or that of its P3 adjoint's spectrum, which goes with its cube)
is below the smallest normal float, beside brighter neighbours."""
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


def _adjoint_errors(x, g):
    """Largest difference of each column of a stack's adjoint from its own
    one-column call, and that call's largest entry."""
    eng = tta.engine_for(torch.device("cuda", 0))
    pf = [(3, -1, -1)]
    got = eng.circus_backward(x, pf, g)[0].double()
    one = torch.stack([eng.circus_backward(x[:, c:c + 1].contiguous(), pf,
                                           g[:, :, c:c + 1].contiguous())[0, 0]
                       for c in range(x.shape[1])]).double()
    return (got - one).abs().amax(-1), one.abs().amax(-1)


# both are float transforms of the column: within 1e-4 of its largest entry, as
# the pairs of ordinary columns are held to
@pytest.mark.parametrize("rows", [363, 1267])
@pytest.mark.parametrize("factor", [1e-6, 2.5e-7, 1e-7, 5e-8, 2e-8, 1e-8, 1e-9])
def test_adjoint_dim_column_beside_a_bright_one(rows, factor):
    x = _columns(rows, 4, 9)
    x[0, 1] *= factor
    x[0, 2] *= factor
    err, top = _adjoint_errors(x, torch.ones((1, 1, 4), device="cuda"))
    assert torch.all(top > 0) and torch.all(err <= 1e-4 * top), (err / top).tolist()


@pytest.mark.parametrize("rows", [363, 1267])
@pytest.mark.parametrize("ratio", [0.9, 0.6, 0.1])
def test_adjoint_dim_neighbours(rows, ratio):
    """Two neighbours dimmed together, over the scales at which the squared norms
    of their spectra pass the smallest normal float one after the other."""
    scales = np.geomspace(1e-6, 3e-9, 26)
    x = _columns(rows, 1, 4).repeat(1, 2 * len(scales), 1)
    for i, s in enumerate(scales):
        x[0, 2 * i] *= s
        x[0, 2 * i + 1] *= ratio * s
    err, top = _adjoint_errors(x, torch.ones((1, 1, x.shape[1]), device="cuda"))
    assert torch.all(top > 0) and torch.all(err <= 1e-4 * top), (err / top).tolist()


@pytest.mark.parametrize("factor", [1e-19, 1e-22, 1e-24, 1e-25, 1e-26, 1e-27])
def test_p3_dim_column_beside_a_bright_one(factor):
    """|F / n|^4 of such a column underflows: zero, whatever its neighbour is."""
    eng = tta.engine_for(torch.device("cuda", 0))
    x = _columns(2101, 4, 7)
    bright = eng.circus(x, [(3, -1, -1)])[0, 0]
    x[0, 1] *= factor
    x[0, 2] *= factor
    got = eng.circus(x, [(3, -1, -1)])[0, 0]
    assert got[1] == 0 and got[2] == 0
    # one more or one fewer column in the transform: the float FFT's 1.4e-5
    assert torch.allclose(got[[0, 3]], bright[[0, 3]], rtol=2.8e-5, atol=0)
