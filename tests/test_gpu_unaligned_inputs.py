"""Inputs that are contiguous views off the 16-byte grid of the kernels' wide loads: the Python functions
copy them, the C entry points refuse them, nothing reads them misaligned."""

import pytest
import torch

from helpers import gen

pytestmark = pytest.mark.gpu


def shifted(t, by=1):
    flat = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    flat[by:] = t.reshape(-1)
    return flat[by:].view(t.shape)


@pytest.mark.parametrize("k", [64, 336])
def test_second_moment_at_any_float(k):
    from hi2_b200 import _lib
    from hi2_b200.hessian import transform_sigma

    x = torch.randn(2 * k, k, generator=gen(k))
    sigma, had = (x.T @ x).cuda(), torch.ones(k // 16, dtype=torch.uint8)
    view = shifted(sigma)
    assert view.is_contiguous() and view.data_ptr() % 16 == 4
    assert torch.equal(transform_sigma(view, None, had, 2.0), transform_sigma(sigma, None, had, 2.0))
    hs = torch.empty(k, k, device="cuda")
    for a, b in ((view, hs), (sigma, shifted(hs))):
        with pytest.raises(ValueError, match="aligned"):
            _lib.call("hi2_transform_sigma_host_flags", _lib.ptr(a), 1.0, None, _lib.ptr(had), k, _lib.ptr(b), None,
                      _lib.stream(sigma.device))
