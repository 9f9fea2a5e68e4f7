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


@pytest.mark.parametrize("k,nbits", [(192, (2, 4)), (640, (2, 4)), (640, (8, 8))])  # FMA, tensor-core and FMA updates
def test_factor_at_any_float(k, nbits):
    from hi2_b200 import _lib
    from hi2_b200.hessian import GptqJob, encode_jobs_gptq

    g = gen(k)
    u = (torch.triu(torch.randn(k, k, generator=g) * 0.02) + torch.eye(k)).cuda()
    w, d = (torch.randn(200, k, generator=g) * 0.02).cuda(), torch.ones(k, device="cuda")
    view = shifted(u)

    def encoded(factor):
        return encode_jobs_gptq([GptqJob(w[:70], d, factor, nbits[0], 32), GptqJob(w[70:], d, factor, nbits[1], 32)], "fast")

    for a, b in zip(encoded(view), encoded(u)):
        assert torch.equal(a.codes, b.codes) and torch.equal(a.params, b.params)
    rows, cols = 16, torch.arange(k, device="cuda", dtype=torch.int32)
    codes, lo = torch.empty(rows, k, dtype=torch.uint8, device="cuda"), torch.zeros(rows, k // 16, device="cuda")
    ptrs = torch.tensor([u.data_ptr()], device="cuda")  # what the kernel would read: the aligned one
    with pytest.raises(ValueError, match="aligned"):
        _lib.call("hi2_gptq_round", _lib.ptr(w), rows, k, _lib.ptr(torch.empty(rows, 128, device="cuda")), _lib.ptr(codes),
                  _lib.ptr(lo), _lib.ptr(lo), k // 16, _lib.ptr(torch.zeros(rows, dtype=torch.int32, device="cuda")),
                  _lib.ptr(ptrs), _lib.ptr(cols // 32), _lib.ptr(torch.ones(1, device="cuda")), None, 1,
                  _lib.host_i64([0, rows]), _lib.host_i64([view.data_ptr()]), _lib.stream(w.device))
