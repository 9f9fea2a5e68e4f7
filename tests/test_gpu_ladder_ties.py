"""The ladder search where a column lies on, or within rounding of, the middle between two levels, on
blocks shared by two lanes, and on steps outside the range of the reciprocal: bit for bit the oracle."""

import pytest
import torch

from helpers import gen
from oracle import ptq_oracle as po

pytestmark = pytest.mark.gpu


def block(kind, rows, k, seed):
    g = gen(seed)
    if kind == "levels":  # every value a level or the middle between two, for many of the ladders tried
        w = torch.randint(-6, 7, (rows, k), generator=g).float() / 2
    elif kind == "near":  # a few ulp either side of such a middle
        w = torch.randint(-6, 7, (rows, k), generator=g).float() / 2
        w = w * (1 + torch.randint(-3, 4, (rows, k), generator=g).float() * 2.0**-23)
    elif kind == "offset":  # a ladder far from zero: every sum x_hat - x cancels
        w = 100 + torch.randn(rows, k, generator=g) * 0.02
    elif kind == "constant":
        w = torch.full((rows, k), 0.37)
    elif kind == "tiny":
        w = torch.randn(rows, k, generator=g) * 1e-20
    else:
        w = torch.randn(rows, k, generator=g)
    return w


@pytest.mark.parametrize("kind", ["levels", "near", "offset", "constant", "tiny", "plain"])
@pytest.mark.parametrize("n", [2, 4, 16, 256])
@pytest.mark.parametrize("b", [16, 32, 64])
def test_search_on_ties(kind, n, b):
    from hi2_b200.encode import fit_ladder

    for rows, effort in ((1, "normal"), (15, "max"), (17, "fast"), (33, "normal")):
        w = block(kind, rows, 192, 7 * n + b + rows).reshape(rows, 192 // b, b)
        d = (0.1 + torch.rand(1, 192 // b, b, generator=gen(rows)))
        lo, st = fit_ladder(w.cuda(), d.cuda(), n, effort)
        want = po.search_ladder(w, d, n, effort)
        assert torch.equal(lo.cpu(), want[0]) and torch.equal(st.cpu(), want[1])
