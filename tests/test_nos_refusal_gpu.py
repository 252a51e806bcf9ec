"""Orthonormal calls that are refused leave the plan's device buffers as they
were (the captured graphs of the calls that are not hold their addresses)."""
import numpy as np
import pytest
import torch

from tracetransform_gb300._native import TTError
from tracetransform_gb300.device import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,message", [(9001, 1000, "aligned rows exceeds"),
                                               (7000, 1025, "exceeds 1024"),
                                               (600, 2000, "at least as many rows")])
def test_refusal_keeps_the_buffers(rows, cols, message):
    eng = Engine(0)
    rng = np.random.default_rng(1)
    good = torch.from_numpy(rng.random((2, 64, 300)).astype(np.float32)).cuda()
    bad = torch.from_numpy(rng.random((1, cols, rows)).astype(np.float32)).cuda()
    out = torch.empty((2, 1, 64), device="cuda")
    refused = torch.empty((1, 1, cols), device="cuda")
    eng.circus_orthonormal(good, [1], out=out)
    # the medians' own buffer, which every call fills, at the refused call's size
    eng.circus_orthonormal(good.repeat(20, 1, 1), [1])
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    with pytest.raises(TTError, match=message):
        eng.circus_orthonormal(bad, [1], out=refused)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free0
    again = torch.empty_like(out)
    eng.circus_orthonormal(good, [1], out=again)
    assert torch.equal(out, again)
