"""Orthonormal calls whose buffers fit the device only at the call's own size, not at
that of the longest columns of its row class."""
import numpy as np
import pytest
import torch

from tracetransform_gb300 import _native
from tracetransform_gb300.device import Engine

pytestmark = pytest.mark.gpu


def test_own_size_when_the_class_does_not_fit():
    """The refused allocation is the first of a call whose other buffers are there."""
    lib = _native.lib()
    rng = np.random.default_rng(2)
    short, longer = (torch.from_numpy(rng.random((2, 64, rows)).astype(np.float32)).cuda()
                     for rows in (300, 600))
    want, centers = Engine(0).circus_orthonormal(longer, [1, 2])
    eng = Engine(0)
    eng.circus_orthonormal(short, [1])
    assert lib.tt_debug_fail_allocations(1) == 0
    try:
        got, c = eng.circus_orthonormal(longer, [1, 2])
    finally:
        lib.tt_debug_fail_allocations(0)
    assert torch.equal(got, want) and np.array_equal(c, centers)
    got, _ = eng.circus_orthonormal(longer, [1, 2])
    assert torch.equal(got, want)


def test_two_refusals_are_out_of_memory():
    lib = _native.lib()
    sino = torch.rand((2, 64, 600), device="cuda")
    eng = Engine(0)
    eng.circus_orthonormal(sino[:, :, :300].contiguous(), [1])
    assert lib.tt_debug_fail_allocations(2) == 0
    try:
        with pytest.raises(_native.TTError) as e:
            eng.circus_orthonormal(sino, [1])
        assert e.value.status == 5
    finally:
        lib.tt_debug_fail_allocations(0)
    out, _ = eng.circus_orthonormal(sino, [1])
    assert torch.isfinite(out).all()
