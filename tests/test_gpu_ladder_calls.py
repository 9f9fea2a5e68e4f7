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


@pytest.mark.parametrize("block,nb", [(16, 262145), (16, 400001), (32, 262145), (64, 262141)])
def test_more_blocks_in_a_row_than_one_grid_dimension_holds(block, nb):
    """Four blocks of a row go to a thread block, and a grid dimension ends at 65535."""
    from hi2_b200.encode import fit_ladder

    wb = torch.randn(1, nb, block, generator=gen(nb))
    db = torch.rand(1, nb, block, generator=gen(block)) + 0.1
    lo, st = fit_ladder(wb.cuda(), db.cuda(), 4, "fast")
    want = po.search_ladder(wb, db, 4, "fast")
    assert torch.equal(lo.cpu(), want[0]) and torch.equal(st.cpu(), want[1])


@pytest.mark.parametrize("block", [16, 32, 64])
@pytest.mark.parametrize("n", [2**22, 2**23, 2**23 + 1, 2**23 + 2, 2**24])
def test_more_levels_than_the_shifted_rounding_covers(block, n):
    """Codes up to 2^23 stay whole numbers after 2^23 is added to them, larger ones do not."""
    from hi2_b200.encode import fit_ladder

    wb = torch.randn(33, 12, block, generator=gen(block))
    db = torch.rand(1, 12, block, generator=gen(n % 1000)) + 0.1
    lo, st = fit_ladder(wb.cuda(), db.cuda(), n, "normal")
    want = po.search_ladder(wb, db, n, "normal")
    assert torch.equal(lo.cpu(), want[0]) and torch.equal(st.cpu(), want[1])
