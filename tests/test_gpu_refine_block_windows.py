"""The refinement block kernel over one to eight windows of columns and one or two rows per lane, against
the column-by-column loop in the same arithmetic: equal bits."""

import pytest
import torch

from helpers import gen

pytestmark = pytest.mark.gpu


def case(rows, k, seed):
    g = gen(seed)
    x = torch.randn(2 * k, k, generator=g)
    hs = (x.T @ x / x.shape[0]).contiguous()
    st = (0.01 + 0.02 * torch.rand(rows, k, generator=g)).half().float()
    lo = (-0.05 * torch.rand(rows, k, generator=g)).half().float()
    st[:, 5] = 0.0
    top = torch.tensor([1.0, 3.0, 15.0, 255.0])[torch.randint(0, 4, (rows,), generator=g)]
    c = torch.floor(torch.rand(rows, k, generator=g) * (top[:, None] + 1)).minimum(top[:, None])
    g_all = 0.02 * torch.randn(rows, k, generator=g)
    return g_all, c, lo, st, top, hs


def column_loop(g_all, c, lo, st, top, hs, b0, length):
    seg, c, dw = g_all[:, b0 : b0 + length].clone(), c.clone(), torch.zeros(c.shape[0], length)
    for i in range(length):
        j = b0 + i
        now = (lo[:, j] + c[:, j] * st[:, j]).half().float()
        gains, moves = [], []
        for sign in (1.0, -1.0):
            q = c[:, j] + sign
            d = (lo[:, j] + q * st[:, j]).half().float() - now
            ok = (q >= 0) & (q <= top) & (st[:, j] > 0)
            gains.append(torch.where(ok, -((2 * d) * seg[:, i] + (d * d) * hs[j, j]), torch.tensor(-torch.inf)))
            moves.append(d)
        minus = gains[1] > gains[0]
        take = torch.where(minus, gains[1], gains[0]) > 0
        dw[:, i] = torch.where(take, torch.where(minus, moves[1], moves[0]), torch.tensor(0.0))
        c[:, j] += torch.where(take, torch.where(minus, torch.tensor(-1.0), torch.tensor(1.0)), torch.tensor(0.0))
        seg[:, i + 1 :] += dw[:, i : i + 1] * hs[j, j + 1 : b0 + length]
    return c, dw


@pytest.mark.parametrize("length", [16, 32, 48, 80, 96, 112, 128])
@pytest.mark.parametrize("rows", [1, 31, 33, 150])
def test_block_against_the_column_loop(length, rows):
    from hi2_b200 import refine_kernel

    g_all, c, lo, st, top, hs = case(rows, 160, length + rows)
    want_c, want_dw = column_loop(g_all, c, lo, st, top, hs, 32, length)
    dev = [t.cuda() for t in (g_all[:, 32 : 32 + length].contiguous(), c, lo, st, top, hs)]
    dw = torch.zeros(rows, length, device="cuda")
    refine_kernel.refine_block(dev[0], dev[1], *dev[2:], 32, length, dw)
    assert torch.equal(dev[1].cpu(), want_c) and torch.equal(dw.cpu(), want_dw)


@pytest.mark.parametrize("rows", [18945, 28417])
def test_rows_per_lane_do_not_change_anything(rows):
    from hi2_b200 import refine_kernel

    g_all, c, lo, st, top, hs = [t.cuda() for t in case(rows, 128, rows)]
    whole, dw = c.clone(), torch.zeros(rows, 128, device="cuda")
    refine_kernel.refine_block(g_all, whole, lo, st, top, hs, 0, 128, dw)
    for r0 in (0, rows - 1000):
        at = slice(r0, r0 + 1000)
        part, dwp = c[at].clone(), torch.zeros(1000, 128, device="cuda")
        refine_kernel.refine_block(g_all[at].contiguous(), part, lo[at].contiguous(), st[at].contiguous(), top[at].contiguous(), hs,
                                   0, 128, dwp)
        assert torch.equal(whole[at], part) and torch.equal(dw[at], dwp)
