"""The GPTQ block kernel where its mapping changes: block lengths of one to eight windows, one and
two rows per lane, thread blocks whose rows read several factors, and launches shared by neighbouring
units with one factor.  Same inputs, same arithmetic: everything is compared bit for bit."""

import pytest
import torch

from helpers import gen

pytestmark = pytest.mark.gpu


def case(rows, k, groups, seed, nbits=(2, 4, 8)):
    g = gen(seed)
    wc = torch.randn(rows, k, generator=g) * 0.02
    us = [torch.triu(torch.randn(k, k, generator=g) * 0.05) + torch.eye(k) * (0.5 + torch.rand(k, generator=g)) for _ in range(groups)]
    us[0][3, 3] = 1.0 - 2.0**-24  # a pivot whose significand is all ones: no usable reciprocal
    lo, st = -0.04 - 0.01 * torch.rand(rows, k // 16, generator=g), 0.005 + 0.02 * torch.rand(rows, k // 16, generator=g)
    lo, st = lo.half().float(), st.half().float()
    st[::7, 0] = 0.0
    grp = torch.randint(0, groups, (rows,), generator=g).to(torch.int32)
    blk = torch.stack([torch.randint(0, k // 16, (k,), generator=g) for _ in range(groups)]).to(torch.int32)
    nmax = torch.tensor([2.0 ** nbits[i % len(nbits)] - 1 for i in range(groups)])
    return wc, us, lo, st, grp, blk, nmax


def column_loop(wc, us, lo, st, grp, blk, nmax, i1, length):
    """The block one column at a time on the CPU, every operation rounded on its own."""
    seg = wc[:, i1 : i1 + length].clone()
    u = torch.stack(us)[grp.long()][:, i1 : i1 + length, i1 : i1 + length]
    codes, err, comp = torch.zeros_like(seg), torch.zeros_like(seg), torch.zeros_like(seg)
    rows = torch.arange(wc.shape[0])
    for i in range(length):
        b = blk[grp.long(), i1 + i].long()
        l, s, col = lo[rows, b], st[rows, b], seg[:, i].clone()
        q = torch.round((col - l) / torch.where(s == 0, 1.0, s)).clamp_min(0).minimum(nmax[grp.long()])
        q = torch.where(s == 0, 0.0, q)
        e = (col - (l + q * s).half().float()) / u[:, i, i]
        seg[:, i + 1 :] -= e[:, None] * u[:, i, i + 1 :]
        codes[:, i], err[:, i], comp[:, i] = q, e, col
    return codes.to(torch.uint8), err, comp


def block(args, i1, length, comp=True):
    from hi2_b200 import gptq_kernel

    wc, us, lo, st, grp, blk, nmax = args
    dev = "cuda"
    rows, k = wc.shape
    u = [x.to(dev) for x in us]
    codes = torch.zeros(rows, k, dtype=torch.uint8, device=dev)
    err = torch.zeros(rows, length, device=dev)
    seen = torch.zeros(rows, k, device=dev) if comp else None
    gptq_kernel.gptq_block(wc.to(dev), i1, length, err, codes, lo.to(dev), st.to(dev), grp.to(dev),
                           torch.tensor([x.data_ptr() for x in u], device=dev), blk.to(dev), nmax.to(dev), seen)
    torch.cuda.synchronize()
    return codes[:, i1 : i1 + length].cpu(), err.cpu(), seen[:, i1 : i1 + length].cpu() if comp else None


@pytest.mark.parametrize("length", [16, 32, 48, 64, 80, 96, 112, 128])
@pytest.mark.parametrize("rows,groups", [(1, 1), (31, 1), (33, 2), (200, 3)])
def test_block_against_the_column_loop(length, rows, groups):
    args = case(rows, 160, groups, 31 * length + rows)
    codes, err, comp = column_loop(*args, 32, length)
    got = block(args, 32, length)
    assert torch.equal(got[0], codes) and torch.equal(got[1], err) and torch.equal(got[2], comp)
    plain = block(args, 32, length, comp=False)
    assert torch.equal(plain[0], codes) and torch.equal(plain[1], err)


@pytest.mark.parametrize("rows", [18944, 18945, 19007, 28416, 28417])
def test_rows_per_lane_do_not_change_anything(rows):
    args = case(rows, 128, 2, rows)
    whole = block(args, 0, 128)
    for r0 in (0, 9000, rows - 1500):
        part = slice(r0, r0 + 1500)
        wc, us, lo, st, grp, blk, nmax = args
        got = block((wc[part], us, lo[part], st[part], grp[part], blk, nmax), 0, 128)
        for a, b in zip(whole, got):
            assert torch.equal(a[part], b)


@pytest.mark.parametrize("nbits", [(2, 4), (8, 8)])  # tensor-core and FMA trailing updates
def test_units_of_one_factor_share_a_launch_and_nothing_else(nbits):
    """Jobs with one factor next to each other give what each of them gives alone."""
    from hi2_b200.hessian import GptqJob, encode_jobs_gptq

    k = 640
    w, us, *_ = case(700, k, 2, 5)
    w, us, d = w.cuda(), [u.cuda() for u in us], torch.ones(k, device="cuda")
    cuts = [(0, 130, 0, nbits[0]), (130, 131, 0, nbits[1]), (131, 400, 0, nbits[0]), (400, 533, 1, nbits[1]), (533, 700, 0, nbits[1])]
    jobs = [GptqJob(w[a:b].contiguous(), d, us[f], nb, 32) for a, b, f, nb in cuts]
    for job, got in zip(jobs, encode_jobs_gptq(jobs, "fast", comp=True)):
        alone = encode_jobs_gptq([job], "fast", comp=True)[0]
        assert torch.equal(got.codes, alone.codes) and torch.equal(got.comp, alone.comp) and torch.equal(got.params, alone.params)


@pytest.mark.parametrize("k", [640, 1024, 1040, 1536, 2064])
@pytest.mark.parametrize("rows", [40, 300])
def test_updates_taken_together_are_the_updates_one_by_one(rows, k):
    """One pass over the columns behind a group of blocks adds in the order of the blocks."""
    from hi2_b200 import _lib
    from hi2_b200.gptq_kernel import split_tf32_transposed

    g = gen(rows + k)
    u = [(torch.triu(torch.randn(k, k, generator=g) * 0.02) + torch.eye(k)).cuda() for _ in range(2)]
    split = [split_tf32_transposed(x) for x in u]
    cut = rows // 3
    w = (torch.randn(rows, k, generator=g) * 0.02).cuda()
    lo = (-0.04 - 0.01 * torch.rand(rows, k // 16, generator=g)).half().float().cuda()
    st = (0.005 + 0.02 * torch.rand(rows, k // 16, generator=g)).half().float().cuda()
    grp = (torch.arange(rows) >= cut).to(torch.int32).cuda()
    ptrs = torch.tensor([x.data_ptr() for x in u]).cuda()
    blk = (torch.arange(k) // 32).to(torch.int32).expand(2, k).contiguous().cuda()
    nmax = torch.tensor([3.0, 15.0]).cuda()

    def run(name, *scratch):
        wc, codes, comp = w.clone(), torch.zeros(rows, k, dtype=torch.uint8, device="cuda"), torch.zeros(rows, k, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call(name, _lib.ptr(wc), rows, k, *scratch, _lib.ptr(codes), _lib.ptr(lo), _lib.ptr(st), k // 16, _lib.ptr(grp),
                  _lib.ptr(ptrs), _lib.ptr(blk), _lib.ptr(nmax), _lib.ptr(comp), 2, _lib.host_i64([0, cut, rows]),
                  _lib.host_i64([x.data_ptr() for x in split]), _lib.ptr(status), _lib.stream(w.device))
        assert int(status.item()) == 0
        return codes, comp, wc

    one, parts = torch.empty(rows, 128, device="cuda"), torch.empty(2, rows, 128, device="cuda")
    want = run("hi2_gptq_round_tc", _lib.ptr(one), _lib.ptr(parts))
    for columns in (128, 256, 512, 1024):
        scratch = torch.empty(2, rows, columns, device="cuda")
        got = run("hi2_gptq_round_tc_grouped", _lib.ptr(scratch), columns)
        for a, b in zip(got, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows", [18945, 19007])
@pytest.mark.parametrize("columns", [128, 512])
@pytest.mark.parametrize("with_comp", [False, True])
def test_loop_of_many_rows_is_the_loop_of_a_few(rows, columns, with_comp):
    """Two rows per lane with the errors left as TF32 parts, in a buffer of one block's width and of a
    group's: every row as in a launch of a few hundred rows, one per lane."""
    from hi2_b200 import _lib
    from hi2_b200.gptq_kernel import split_factor

    k, cut = 656, 7001
    wc, us, lo, st, _, _, _ = case(rows, k, 2, rows, (2, 4))
    blk = (torch.arange(k) // 32).to(torch.int32).expand(2, k).contiguous().cuda()
    grp = (torch.arange(rows) >= cut).to(torch.int32).cuda()
    w, lo, st, nmax = wc.cuda(), lo.cuda(), st.cuda(), torch.tensor([3.0, 15.0]).cuda()
    u = [x.cuda() * 0.5 for x in us]
    split, ptrs = [split_factor(x) for x in u], torch.tensor([x.data_ptr() for x in u]).cuda()

    def run(r0, r1):
        n, at = r1 - r0, slice(r0, r1)
        work, codes = w[at].clone(), torch.zeros(n, k, dtype=torch.uint8, device="cuda")
        seen = torch.zeros(n, k, device="cuda") if with_comp else None
        scratch, status = torch.empty(2, n, columns, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        inner = min(max(cut - r0, 0), n)
        lo_r, st_r, grp_r = lo[at].contiguous(), st[at].contiguous(), grp[at].contiguous()
        _lib.call("hi2_gptq_round_tc_grouped", _lib.ptr(work), n, k, _lib.ptr(scratch), columns, _lib.ptr(codes), _lib.ptr(lo_r),
                  _lib.ptr(st_r), k // 16, _lib.ptr(grp_r), _lib.ptr(ptrs), _lib.ptr(blk), _lib.ptr(nmax), _lib.ptr(seen), 2,
                  _lib.host_i64([0, inner, n]), _lib.host_i64([x.data_ptr() for x in split]), _lib.ptr(status),
                  _lib.stream(w.device))
        assert int(status.item()) == 0
        return [codes, work] + ([seen] if with_comp else [])

    whole = run(0, rows)
    for r0, r1 in ((0, 300), (cut - 100, cut + 150), (rows - 333, rows)):
        for a, b in zip(whole, run(r0, r1)):
            assert torch.equal(a[r0:r1], b)


@pytest.mark.parametrize("k", [4, 64, 68, 128, 1040])
def test_split_of_the_factor_where_the_updates_read_it(k):
    from hi2_b200.gptq_kernel import split_factor, split_tf32_transposed

    u = torch.triu(torch.randn(k, k, generator=gen(k))).cuda()
    low = torch.ones(k, k, dtype=torch.bool, device="cuda").tril()
    for got, want in zip(split_factor(u), split_tf32_transposed(u)):
        assert torch.equal(got[low], want[low])
