"""Calls of the ladder search at the edges of what it accepts: bit for bit the oracle."""

import pytest
import torch

from helpers import gen
from oracle import ptq_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 2, 3, 5])
@pytest.mark.parametrize("n", [4, 16])
@pytest.mark.parametrize("block", [16, 32, 64])
def test_weights_may_start_at_any_float(block, n, offset):
    """Column weights that are a contiguous view into a larger buffer, off its grid of 16 bytes."""
    from hi2_b200 import ladder_kernel
    from hi2_b200.encode import EFFORT

    nb, grid = 9, EFFORT["fast"]["grid"]
    wb = torch.randn(33, nb, block, generator=gen(block + n))
    flat = (torch.rand(nb * block + offset, generator=gen(offset)) + 0.1).cuda()
    db = flat[offset:].view(nb, block)
    assert db.is_contiguous() and db.data_ptr() % 16 == 4 * offset % 16
    got = ladder_kernel.ladder_grid(wb.cuda(), db, grid, n)
    for a, b, want in zip(got, ladder_kernel.ladder_grid(wb.cuda(), db.clone(), grid, n),
                          po.grid_search(wb, db.cpu().reshape(1, nb, block), n, grid)):
        assert torch.equal(a, b) and torch.equal(a.cpu(), want)
