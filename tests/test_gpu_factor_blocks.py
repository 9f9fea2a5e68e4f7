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
    # Conditions of H + lam I here: 1 to 3e4.  Measured over these sizes: 0.4 to 2.1 times 2^-24, growing with
    # the reductions, while the products are fp32 chains of at most 288 values, and 5.0 where the two
    # largest of them run on the tensor cores (k = 2048, 2304).  Four times that.
    rel = (u.double() - want).norm() / want.norm()
    tensor_cores = k in (2048, 2304)
    assert rel < (20 if tensor_cores else 4 * (1 + k / 1500)) * 2.0**-24, rel * 2.0**24
    # U^T U (H + lam I) = I ties the result to the input and not to the other solver.  Measured: at most 52
    # times 2^-24 (k = 640, the largest condition), 72 with tensor-core products.
    a = hs.double() + 0.01 * hs.double().diagonal().mean() * torch.eye(k, dtype=torch.float64)
    eye = u.double().T @ u.double() @ a
    worst = (eye - torch.eye(k, dtype=torch.float64)).abs().max()
    assert worst < 4 * (72 if tensor_cores else 52) * 2.0**-24, worst * 2.0**24


def factor(hs, lam=0.0):
    """``(U, info)`` of one attempt, damping ``lam`` itself added to the diagonal."""
    from hi2_b200 import _lib

    hs, k = hs.cuda(), hs.shape[0]
    ws = torch.empty(_lib.load().hi2_inverse_factor_workspace_bytes(k), dtype=torch.uint8, device="cuda")
    u, lam = torch.empty(k, k, device="cuda"), torch.full((1,), lam, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("hi2_inverse_factor", _lib.ptr(hs), _lib.ptr(lam), k, _lib.ptr(u), _lib.ptr(ws), ws.numel(), _lib.ptr(info),
              _lib.stream(hs.device))
    return u.cpu(), int(info.item())


def rounded_once(got, want):
    """fp32 ``got`` is fp64 ``want`` rounded to nearest, but for an error of 1e-13 of the value in what
    was rounded: far above the few ulp (1e-16) of fp64 arithmetic, and so far below fp32's ulp (6e-8)
    that an error of 1e-9 before the rounding would show in one value of a hundred."""
    ulp = torch.ldexp(torch.ones_like(want), torch.frexp(want)[1] - 24)
    return bool(((got.double() - want).abs() <= 0.5 * ulp + 1e-13 * want.abs()).all())


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 63, 64, 65, 100, 127, 128, 129, 300, 2304])
def test_diagonal_inputs_of_every_magnitude(k):
    """U is 1 / sqrt(v) on the diagonal: the reciprocal roots alone, formed in fp64 and rounded once."""
    for seed in range(20 if k < 2000 else 1):
        g = gen(100 * k + seed)
        v = torch.ldexp(1 + torch.rand(k, generator=g), torch.randint(-120, 121, (k,), generator=g))
        u, info = factor(torch.diag(v))
        assert info == 0 and torch.equal(u, torch.diag(u.diagonal()))
        assert rounded_once(u.diagonal(), 1 / v.double().sqrt())


@pytest.mark.parametrize("k,bad", [(1, 0), (8, 0), (8, 7), (64, 30), (128, 5), (200, 199)])
@pytest.mark.parametrize("value", [0.0, -1.0, -1e-30, float("nan")])
def test_a_bad_pivot_counts_as_one_and_its_neighbours_stay(k, bad, value):
    """The eight columns around a bad pivot take the plain root and quotient one by one."""
    g = gen(k + bad)
    v = torch.ldexp(1 + torch.rand(k, generator=g), torch.randint(-60, 61, (k,), generator=g))
    h = torch.diag(v)
    h[bad, bad] = value
    u, info = factor(h)
    want = 1 / v.double().sqrt()
    want[bad] = 1.0
    assert info == (k - 1 - bad) + 1
    assert torch.equal(u, torch.diag(u.diagonal())) and rounded_once(u.diagonal(), want)


@pytest.mark.parametrize("k,bad", [(100, 70), (300, 290), (400, 10)])
def test_pivot_index_of_an_indefinite_input(k, bad):
    """The reversed matrix meets the bad pivot where the identity turns negative."""
    hs = torch.eye(k)
    hs[bad, bad] = -1.0
    assert factor(hs)[1] == (k - 1 - bad) + 1
