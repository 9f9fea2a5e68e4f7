"""Local code refinement after GPTQ on B200 (interface of hi2/refine.py:24-162).

A sweep visits the columns in blocks of 128: one launch of the block kernel decides every column
of the block for every row (csrc/refine.cu), one fp32-grade product (three TF32 tcgen05 products,
csrc/lazy_tc.cu; fp32 FMA for narrow inputs and 256-level rows) brings ``g = e Hs`` up to date for
the other columns.  Ladders are never touched.
"""

from __future__ import annotations

import torch

from . import _lib, refine_kernel
from .format import decode_params

BLOCK_COLUMNS = 128
GROUP_BLOCKS = 4  # blocks whose moves reach the far columns of g in one product
# Rows x columns from which grouping pays (below, a step is a latency chain).  Two sweeps at K = 4096, a block at
# a time / groups of four, ms: 2048 rows 2.78 / 3.61, 4096 rows 3.83 / 4.44, 6144 rows 5.57 / 5.55, 8192 rows
# (the line) 6.69 / 6.27, 11008 rows 9.02 / 8.02; 1024 x 11008 8.40 / 10.6, 4096 x 8192 11.9 / 11.6, 4096 x 11008
# 20.5 / 18.5.  Groups of two or eight blocks are no better on either side.
GROUP_MIN_ELEMS = 1 << 25
TC_MIN_K = 512  # inputs at least this wide take the tensor-core products


@torch.no_grad()
def objective(w, codes, lo, step, hs, block) -> float:
    """Sum over rows of ``e Hs e^T`` for the decoded codes."""
    idx = torch.arange(w.shape[1], device=w.device) // block
    e = ((lo[:, idx] + codes.float() * step[:, idx]).half().float() - w).contiguous()
    g = torch.empty_like(e)
    refine_kernel.gemm(e, hs.float().contiguous(), g)
    return float((g * e).sum())


def _expand(lo: torch.Tensor, step: torch.Tensor, block: int):
    """Per-column ladders ``[N, K]`` from the per-block ones ``[N, K / block]``."""
    return lo.repeat_interleave(block, dim=1), step.repeat_interleave(block, dim=1)


def _use_tc(use_tc: bool, k: int) -> bool:
    """The two products of a sweep, g = e Hs and g += dw Hs[b0:b1], run on the tensor cores as three TF32
    products (fp32-grade; Hs is symmetric, so its rows are the K-major right operand as they lie).  Rows
    with 256 levels and narrow inputs keep the fp32 FMA product, as in the GPTQ path."""
    return use_tc and k >= TC_MIN_K and k % 4 == 0


@torch.no_grad()
def _sweeps(w, codes, lo_x, st_x, top, hs, passes: int, use_tc: bool | None, wait: bool):
    """:func:`_run` for rows given with a ladder per column."""
    _lib.need_cuda(w, codes, lo_x, st_x, top, hs)
    c = codes.float().contiguous().clone()
    lo_x, st_x = lo_x.float().contiguous(), st_x.float().contiguous()
    e = [((lo_x + c * st_x).half().float() - w.float()).contiguous()]
    use_tc = _use_tc(bool((top <= 15).all()) if use_tc is None else use_tc, w.shape[1])
    if use_tc:
        e = [refine_kernel.split_tf32(e.pop())]
    return _run(c, lo_x, st_x, top.float().reshape(-1).contiguous(), e, hs.float().contiguous(), passes, use_tc, wait)


@torch.no_grad()
def _run(c, lo_x, st_x, top, e: list, hs, passes: int, use_tc: bool, wait: bool):
    """``(refined codes (float), status word or None)`` from fp32 codes ``c [N, K]`` (changed in place) and
    their errors ``e`` (as TF32 parts with ``use_tc``; a list of one entry, which the caller holds nowhere else:
    it is taken out, and its memory is free again behind the first product).  With ``wait``
    the host follows the device: it stops after a sweep that moved no code and raises on a raised
    status word.  Without, nothing is read back: every sweep is queued (one that moves nothing changes
    nothing) and the status word is left to the caller, so several tensors can be refined side by side
    on streams."""
    dev = _lib.need_cuda(c, lo_x, st_x, top, hs)
    if not refine_kernel.available(dev):
        raise RuntimeError(f"refine kernel unavailable on {dev}: {refine_kernel.failure()}")
    n_rows, k = c.shape
    g = torch.empty(n_rows, k, dtype=torch.float32, device=dev)
    status = hs_split = None
    if use_tc:
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        hs_split = refine_kernel.split_tf32(hs)
        refine_kernel.gemm_tc(e.pop(), hs_split, g, status)
    else:
        refine_kernel.gemm(e.pop(), hs, g)
    # With tensor-core products the block kernel reads its slice of g in place and leaves the changes
    # as TF32 parts, and g is brought up to date lazily, as the GPTQ loop does: after a block only the
    # later blocks of its group of GROUP_BLOCKS need its moves now (a narrow product); the columns
    # outside the group take the moves of the whole group in one product with a reduction of up to
    # 512 (a 128 KiB tile of g is then read and written once per 100 MFLOP instead of once per 25);
    # the group's own columns at or before each block, needed by the next sweep only, follow per
    # column block.  The contributions to every g are the same, in another order.  Few rows make
    # every step a latency chain, where more launches cost more than the better products gain: then
    # a group is one block and its update one product.
    width = (GROUP_BLOCKS if n_rows * k >= GROUP_MIN_ELEMS else 1) * BLOCK_COLUMNS
    moves = torch.empty(*((2, n_rows, min(width, k)) if use_tc else (n_rows, BLOCK_COLUMNS)), dtype=torch.float32, device=dev)
    moved = torch.zeros(1, dtype=torch.int32, device=dev) if wait else None
    for sweep in range(passes):
        last = sweep + 1 == passes  # nobody reads g behind it
        refine_kernel.sweep(g, c, lo_x, st_x, top, hs, hs_split, moves, width, last, moved, status)
        if wait and not last:  # whether the next sweep is worth queueing
            if not int(moved.item()):
                break
            moved.zero_()
    if wait and use_tc and int(status.item()):
        raise RuntimeError("refine: a bounded device-side wait ran out in a tensor-core product")
    return c, status


def refine_expanded(w, codes, lo_x, st_x, top, hs, passes: int) -> torch.Tensor:
    """Refined codes (float) of rows ``w [N, K]`` with per-column ladders ``lo_x``/``st_x`` and
    the highest code of each row ``top [N]``; stops early when a sweep moves no code."""
    return _sweeps(w, codes, lo_x, st_x, top, hs, passes, None, True)[0]


def refine_codes(w, codes, lo, step, hs, nbits: int, block: int, passes: int) -> torch.Tensor:
    """:func:`refine_expanded` for rows rounded at one ``(nbits, block)`` with decoded ladders
    ``lo``/``step [N, K / block]``; returns codes of the dtype of ``codes``."""
    lo_x, st_x = _expand(lo, step, block)
    top = torch.full((w.shape[0],), float(2**nbits - 1), device=w.device)
    return refine_expanded(w, codes, lo_x, st_x, top, hs, passes).to(codes.dtype)


def _decoded(enc):
    lo, step = decode_params(
        enc.params[..., 0], enc.params[..., 1], enc.consts[:, 0:1], enc.consts[:, 1:2],
        enc.consts[:, 2:3],
    )
    return lo.float(), step.float()


def _as_encoded(w, enc, block: int) -> bool:
    """Whether ``enc`` has the types and shapes an encode of this package leaves, which
    :func:`hi2_b200.refine_kernel.prepare` reads."""
    n, k = w.shape
    return (enc.codes.dtype == torch.uint8 and enc.params.dtype == torch.uint8 and enc.consts.dtype == torch.float16
            and block in (16, 32, 64) and k % block == 0 and tuple(enc.codes.shape) == (n, k)
            and tuple(enc.params.shape) == (n, k // block, 2) and tuple(enc.consts.shape) == (n, 3))


def refine_groups(groups, hs: torch.Tensor, passes: int, wait: bool = True):
    """One sweep over the rows of every ``(w, enc, nbits, block)`` group (rows of different
    candidates, and of different tensors that read the same input, share the column loop); returns
    the refined codes per group.  ``wait=False`` reads nothing back and returns ``(codes per group,
    status word or None)``: the caller checks the word once it has queued everything."""
    use_tc = max(g[2] for g in groups) <= 4
    plain = all(_as_encoded(w, enc, block) for w, enc, _, block in groups)
    sizes = [w.shape[0] for w, *_ in groups]
    if plain:  # one pass over each group's rows
        dev = _lib.need_cuda(*[w for w, *_ in groups], hs)
        n, k = sum(sizes), groups[0][0].shape[1]
        use_tc = _use_tc(use_tc, k)
        c, lo_x, st_x = (torch.empty(n, k, dtype=torch.float32, device=dev) for _ in range(3))
        e = [torch.empty(*((2,) if use_tc else ()), n, k, dtype=torch.float32, device=dev)]
        top = torch.empty(n, dtype=torch.float32, device=dev)
        r0 = 0
        for (w, enc, nbits, block), rows in zip(groups, sizes):
            at = slice(r0, r0 + rows)
            wf = w.float()
            if wf.stride(1) != 1 or wf.stride(0) < k or wf.stride(0) % 4 or wf.data_ptr() % 16:
                wf = wf.clone(memory_format=torch.contiguous_format)  # of one row too, whose stride may be anything
            refine_kernel.prepare(wf, _lib.on_grid(enc.codes, 4), _lib.on_grid(enc.params, 2), enc.consts.contiguous(), block, c[at],
                                  lo_x[at], st_x[at], *((e[0][0, at], e[0][1, at]) if use_tc else (e[0][at],)))
            top[at] = float(2**nbits - 1)
            r0 += rows
        out, status = _run(c, lo_x, st_x, top, e, hs.float().contiguous(), passes, use_tc, wait)
    else:
        parts = []
        for w, enc, nbits, block in groups:
            lo, step = _decoded(enc)
            lo_x, st_x = _expand(lo, step, block)
            top = torch.full((w.shape[0],), float(2**nbits - 1), device=w.device)
            parts.append((w.float(), enc.codes.float(), lo_x, st_x, top))
        cat = [torch.cat([p[i] for p in parts]) for i in range(5)]
        out, status = _sweeps(*cat, hs, passes, use_tc, wait)
    codes = [c.to(groups[i][1].codes.dtype) for i, c in enumerate(out.split(sizes))]
    return codes if wait else (codes, status)


def refine_encoded(enc, w, hs, nbits: int, block: int, passes: int):
    """``enc`` with refined codes and a refreshed ``sse`` (weights ``diag(hs)``)."""
    (codes,) = refine_groups([(w, enc, nbits, block)], hs, passes)
    lo, step = _decoded(enc)
    dev = w.device
    k = w.shape[1]
    wf = w.float().contiguous()
    codes = codes.contiguous()
    d = hs.diagonal().float().contiguous()
    lo, step = lo.contiguous(), step.contiguous()
    sse = torch.empty(w.shape[0], dtype=torch.float32, device=dev)
    _lib.call(
        "hi2_ladder_sse", _lib.ptr(codes), _lib.ptr(wf), wf.stride(0), _lib.ptr(d), _lib.ptr(lo),
        _lib.ptr(step), lo.shape[1], w.shape[0], k, block, _lib.ptr(sse), _lib.stream(dev),
    )
    return type(enc)(codes, enc.params, enc.consts, sse, enc.comp)
