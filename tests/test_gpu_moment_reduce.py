"""The sum of item tiles into S at widths that end inside a 64 x 64 piece, a tile, and a diagonal piece, with
one and several splits, on top of an earlier sum, for both tensor-core kernels."""

import pytest
import torch

from helpers import activations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [256, 272, 336, 1024, 1040, 1136, 2064])
@pytest.mark.parametrize("tokens", [300, 8200, 20000])  # below and above the pair kernel's 8192
def test_sum_and_mirror(k, tokens):
    from hi2_b200.hessian import HessianStats

    x = activations(tokens, k, k + tokens, dtype=torch.bfloat16).cuda()
    h = HessianStats(k, "cuda")
    h.update(x)
    first = h.S.clone()
    assert torch.equal(first, first.T)
    exact = x.double().T @ x.double()
    scale = exact.diagonal().sqrt()
    # products are exact in fp32; sums in tensor memory lose at most 2^-23 a step over 1024 tokens
    bound = 1024 / 16 * 2.0**-23
    assert ((first.double() - exact).abs() / (scale[:, None] * scale)).max() < bound
    h.update(x)
    assert torch.equal(h.S, first + first)
