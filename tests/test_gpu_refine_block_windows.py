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


@pytest.mark.parametrize("rows,k", [(1, 64), (3, 192), (70, 1088), (33, 4160)])
@pytest.mark.parametrize("nbits,block", [(2, 16), (4, 64), (8, 32)])
def test_prepare_is_the_elementwise_form(rows, k, nbits, block):
    from hi2_b200 import refine_kernel
    from hi2_b200.encode import encode_rows
    from hi2_b200.refine import _decoded, _expand

    w = torch.randn(rows, k, generator=gen(rows + k)).cuda()
    w[::2, : k // 2] = 0
    enc = encode_rows(w, torch.ones(k, device="cuda"), nbits, block, "fast")
    lo_x, st_x = _expand(*_decoded(enc), block)
    e = (lo_x + enc.codes.float() * st_x).half().float() - w
    c, lo, st, got, low = (torch.empty(rows, k, device="cuda") for _ in range(5))
    refine_kernel.prepare(w, enc.codes, enc.params, enc.consts, block, c, lo, st, got)
    assert torch.equal(c, enc.codes.float()) and torch.equal(lo, lo_x) and torch.equal(st, st_x) and torch.equal(got, e)
    refine_kernel.prepare(w, enc.codes, enc.params, enc.consts, block, c, lo, st, got, low)
    assert torch.equal(torch.stack([got, low]), refine_kernel.split_tf32(e.contiguous()))


@pytest.mark.parametrize("k", [192, 640, 1152])
@pytest.mark.parametrize("width", [128, 512])
@pytest.mark.parametrize("split", [False, True])  # FMA and tensor-core products
def test_last_sweep_leaves_out_only_what_nobody_reads(k, width, split):
    """A sweep that is not followed by another does not bring the columns it has passed up to date: same
    codes, bit for bit, as a sweep that does, and the same word for whether a code moved."""
    from hi2_b200 import refine_kernel

    rows = 90
    g_all, c, lo, st, top, hs = [t.cuda() for t in case(rows, k, k + width)]
    parts = refine_kernel.split_tf32(hs) if split else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for last in (False, True):
        g, codes = g_all.clone(), c.clone()
        moves = torch.empty(*((2, rows, min(width, k)) if split else (rows, 128)), device="cuda")
        moved = torch.zeros(1, dtype=torch.int32, device="cuda")
        refine_kernel.sweep(g, codes, lo, st, top, hs, parts, moves, width, False, moved, status)
        first = codes.clone()
        assert int(moved.item()) == 1 and bool((first != c).any())
        moved.zero_()
        refine_kernel.sweep(g, codes, lo, st, top, hs, parts, moves, width, last, moved, status)
        assert int(moved.item()) == int(bool((codes != first).any())) == 1
        out.append(codes)
    assert torch.equal(*out) and int(status.item()) == 0


@pytest.mark.parametrize("k", [192, 640])  # FMA and tensor-core products
@pytest.mark.parametrize("group", [False, True])
def test_two_sweeps_are_one_and_one(k, group, monkeypatch):
    """Two sweeps in one call give the codes of two sweeps queued one by one from the same start."""
    from hi2_b200 import refine, refine_kernel
    from hi2_b200.encode import encode_rows
    from hi2_b200.refine import refine_groups

    if group:
        monkeypatch.setattr(refine, "GROUP_MIN_ELEMS", 0)
    rows, split = 90, k >= refine.TC_MIN_K
    x = torch.randn(2 * k, k, generator=gen(k))
    hs = (x.T @ x / x.shape[0]).cuda()
    w = torch.randn(rows, k, generator=gen(k + 1)).cuda()
    enc = encode_rows(w, hs.diagonal().contiguous(), 4, 32, "fast")
    c, lo, st, g = (torch.empty(rows, k, device="cuda") for _ in range(4))
    e = torch.empty(2, rows, k, device="cuda") if split else torch.empty(rows, k, device="cuda")
    refine_kernel.prepare(w, enc.codes, enc.params, enc.consts, 32, c, lo, st, *(e if split else (e,)))
    parts, status = refine_kernel.split_tf32(hs) if split else None, torch.zeros(1, dtype=torch.int32, device="cuda")
    if split:
        refine_kernel.gemm_tc(e, parts, g, status)
    else:
        refine_kernel.gemm(e, hs, g)
    width = 512 if group else 128
    moves = torch.empty(*((2, rows, min(width, k)) if split else (rows, 128)), device="cuda")
    top = torch.full((rows,), 15.0, device="cuda")
    for _ in range(2):
        refine_kernel.sweep(g, c, lo, st, top, hs, parts, moves, width, False, None, status)
    assert bool((c != enc.codes).any()) and int(status.item()) == 0
    assert torch.equal(refine_groups([(w, enc, 4, 32)], hs, 2)[0].float(), c)
    codes, word = refine_groups([(w, enc, 4, 32)], hs, 2, False)
    assert torch.equal(codes[0].float(), c) and (word is None or int(word.item()) == 0)


@pytest.mark.parametrize("k", [192, 640])
def test_sweeps_settle(k):
    from hi2_b200.encode import Encoded, encode_rows
    from hi2_b200.refine import refine_groups

    x = torch.randn(2 * k, k, generator=gen(k))
    hs = (x.T @ x / x.shape[0]).cuda()
    w = torch.randn(90, k, generator=gen(k + 1)).cuda()
    enc = encode_rows(w, hs.diagonal().contiguous(), 4, 32, "fast")
    for wait in (True, False):
        many = refine_groups([(w, enc, 4, 32)], hs, 40, wait)
        many = many[0] if wait else many[0][0]
        again = refine_groups([(w, Encoded(many, enc.params, enc.consts, enc.sse), 4, 32)], hs, 1)[0]
        assert (again != many).float().mean() < 1e-3  # after many sweeps nothing moves any more
