"""The rotation adjoint with angles that are no finite number among the others:
such an angle has no lattice, adds nothing, and leaves the others as they are."""
import numpy as np
import pytest
import torch

from tracetransform_gb300.device import Engine

pytestmark = pytest.mark.gpu


def _adjoint(eng, angles, grad):
    """Adjoint of the Radon sinograms of a 40 x 33 image."""
    grad = grad[:, :len(angles)].contiguous()
    med = torch.full(grad.shape, -1, dtype=torch.int32, device="cuda")
    return eng.sinograms_backward(grad, med, 40, 33, angles, [0])


def _grad(n_angles):
    from tracetransform_gb300.api import pad_geometry
    rng = np.random.default_rng(n_angles)
    return torch.from_numpy(
        rng.standard_normal((1, n_angles, pad_geometry(40, 33)[0])).astype(np.float32)).cuda()


# Both forms add the same candidates, each product rounded to 2^-24 of it: a dozen
# terms per angle of at most the largest gradient, far below 1e-5 of the sum.
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 3, 7, 9])
def test_non_finite_angle_adds_nothing(bad, at):
    eng = Engine(0)
    angles = [0, 17, 45, 90, 133, 180, 201, 270, 300, 359]
    grad = _grad(10)
    with_bad = list(angles)
    with_bad[at] = bad
    zeroed = grad.clone()
    zeroed[:, at] = 0
    want = _adjoint(eng, angles, zeroed)
    got = _adjoint(Engine(0), with_bad, grad)
    assert torch.isfinite(got).all()
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert torch.equal(_adjoint(eng, angles, zeroed), want)


def test_all_angles_non_finite():
    eng = Engine(0)
    assert torch.all(_adjoint(eng, [np.nan, np.inf], _grad(2)) == 0)


def test_a_list_with_nan_has_its_own_table():
    """A NaN is neither below nor above any angle: a list holding one must not find
    the table of a list that differs from it there, nor the other way round."""
    angles, nan = [0, 17, 45], [0, np.nan, 45]
    grad = _grad(3)
    first, second = Engine(0), Engine(0)
    want = _adjoint(first, angles, grad)
    zeroed = _adjoint(first, nan, grad)
    assert torch.equal(_adjoint(second, nan, grad), zeroed)
    assert torch.equal(_adjoint(second, angles, grad), want)
    assert not torch.equal(zeroed, want)
