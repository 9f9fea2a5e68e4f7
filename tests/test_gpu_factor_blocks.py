"""The blocked inverse factor at the sizes where its recursion changes shape: inside one leaf of 64,
at the base block of 128, between base blocks, at the products' tiles of 32 and windows of 128, at
the first tensor-core product, and with a leading dimension that needs padding."""

import pytest
import torch

from helpers import gen

pytestmark = pytest.mark.gpu


def damped(k, seed, dead=0):
    x = torch.randn(2 * k + 64, k, generator=gen(seed)) * torch.exp(torch.randn(1, k, generator=gen(seed + 1)))
    if dead:
        x[:, -dead:] = 0.0
    return (x.double().T @ x.double() / x.shape[0]).float()


def exact(hs, damp=0.01):
    a = hs.double()
    a = a + damp * a.diagonal().mean() * torch.eye(a.shape[0], dtype=torch.float64)
    return torch.linalg.inv(torch.linalg.cholesky(a.flip(0, 1))).flip(0, 1)


@pytest.mark.parametrize("k", [1, 3, 7, 16, 63, 64, 65, 80, 127, 128, 129, 144, 160, 192, 193, 255, 256, 272, 384, 400, 513,
                               640, 1000, 1024, 1104, 2032, 2048, 2064, 2304])
def test_factor_against_fp64(k):
    from hi2_b200.hessian import inverse_factor

    hs = damped(k, k)
    u = inverse_factor(hs.cuda(), 0.01).cpu()
    want = exact(hs)
    assert torch.equal(u, u.triu())
    # backward-stable fp32: c * n * eps * cond(L); cond(H + lam I) is below 1e4 here (damping 0.01 of the
    # mean diagonal against a largest eigenvalue of a few dozen means), its root below 1e2, and the sums
    # are cut into pieces of at most 256
    rel = (u.double() - want).norm() / want.norm()
    assert rel < 256 * 2.0**-24 * 1e2 / 10, rel
    # U^T U (H + lam I) = I ties the result to the input and not to the other solver
    a = hs.double() + 0.01 * hs.double().diagonal().mean() * torch.eye(k, dtype=torch.float64)
    eye = u.double().T @ u.double() @ a
    assert (eye - torch.eye(k, dtype=torch.float64)).abs().max() < 1e-2


@pytest.mark.parametrize("k,bad", [(100, 70), (300, 290), (400, 10)])
def test_pivot_index_of_an_indefinite_input(k, bad):
    """The reversed matrix meets the bad pivot where the identity turns negative."""
    from hi2_b200 import _lib

    hs = torch.eye(k, device="cuda")
    hs[bad, bad] = -1.0
    need = _lib.load().hi2_inverse_factor_workspace_bytes(k)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    u, lam = torch.empty(k, k, device="cuda"), torch.zeros(1, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("hi2_inverse_factor", _lib.ptr(hs), _lib.ptr(lam), k, _lib.ptr(u), _lib.ptr(ws), ws.numel(), _lib.ptr(info),
              _lib.stream(hs.device))
    assert int(info.item()) == (k - 1 - bad) + 1
