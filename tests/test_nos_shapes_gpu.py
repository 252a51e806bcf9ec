"""Orthonormal circus at the edges of the QR's row classes, on one plan in turn:
a captured QR must not serve taller columns than it was captured for, and the
results must not depend on what the plan ran before."""
import numpy as np
import pytest
import torch

from tracetransform_gb300.device import Engine

pytestmark = pytest.mark.gpu


def _stack(rows, angles, spreads, seed):
    """One sinogram per spread: bumps whose medians move by up to `spread` rows,
    so that it aligns to about rows + 2 spread."""
    rng = np.random.default_rng(seed)
    t = np.arange(rows)
    out = []
    for spread in spreads:
        mid = rows / 2 + spread * np.sin(np.linspace(0, 2 * np.pi, angles, endpoint=False) * 3)
        x = np.exp(-((t[None] - mid[:, None]) / (rows / 9)) ** 2) + 0.05 * rng.random((angles, rows))
        out.append(x)
    return torch.from_numpy(np.stack(out).astype(np.float32)).cuda()


# aligned rows below, at and above each class limit (512, 1024, 1536, 2048)
SHAPES = [(460, 40, (20, 20)), (470, 40, (30, 2)), (980, 40, (10, 10)), (990, 40, (60, 3)),
          (1500, 40, (10, 10)), (1500, 40, (100, 2)), (2000, 40, (15, 15)), (2000, 40, (120, 1)),
          (460, 40, (20, 20))]


def test_row_classes_on_one_plan():
    shared = Engine(0)
    for k, (rows, angles, spreads) in enumerate(SHAPES):
        sino = _stack(rows, angles, spreads, k)
        got, centers = shared.circus_orthonormal(sino, [1, 2, 3])
        want, wc = Engine(0).circus_orthonormal(sino, [1, 2, 3])
        assert np.array_equal(centers, wc)
        assert torch.equal(got, want), (rows, spreads)
        assert torch.isfinite(got).all()


@pytest.mark.parametrize("rows,angles", [(300, 64), (700, 64), (1300, 64)])
def test_polar_factor_orthonormal(rows, angles):
    """The nearest orthonormal sinogram's columns are orthonormal (float
    rounding of sums over the rows)."""
    from tracetransform_gb300.api import nearest_orthonormal_sinogram
    sino = _stack(rows, angles, (rows // 12,), 3)[0].cpu().numpy().T
    nos, _ = nearest_orthonormal_sinogram(sino)
    g = nos.astype(np.float64).T @ nos.astype(np.float64)
    assert np.abs(g - np.eye(angles)).max() < 1e-5
