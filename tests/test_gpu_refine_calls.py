"""Refinement of encodes and rows whose memory layout differs from what an encode of this package leaves:
strides, alignment and shapes of the inputs do not change the codes."""

import weakref

import pytest
import torch

from helpers import gen

pytestmark = pytest.mark.gpu


def encoded(rows, k, nbits=4, block=32):
    from hi2_b200.encode import encode_rows

    x = torch.randn(2 * k, k, generator=gen(k))
    hs = (x.T @ x / x.shape[0]).cuda()
    w = torch.randn(rows, k, generator=gen(rows)).cuda()
    return w, encode_rows(w, hs.diagonal().contiguous(), nbits, block, "fast"), hs


def shifted(t, by):
    """The values of ``t`` as a contiguous view that starts ``by`` elements into its storage."""
    flat = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    flat[by:] = t.reshape(-1)
    return flat[by:].view(t.shape)


@pytest.mark.parametrize("k", [192, 640])  # FMA and tensor-core products
@pytest.mark.parametrize("kind", ["one row of a wider matrix", "one row repeated", "overlapping rows", "columns one after the other",
                                  "rows off the grid of 16 bytes", "bytes off the grid", "constants with spare columns"])
def test_layout_of_the_inputs_does_not_matter(kind, k):
    from hi2_b200.encode import Encoded
    from hi2_b200.refine import refine_groups

    rows = 1 if kind == "one row of a wider matrix" else 40
    w, enc, hs = encoded(rows, k)
    if kind == "one row of a wider matrix":
        wide = torch.zeros(1, k + 1, device="cuda")
        wide[:, :k] = w
        given = wide[:, :k]
    elif kind == "one row repeated":
        w = w[:1].expand(rows, k)
        given, w = w, w.contiguous()
    elif kind == "overlapping rows":
        flat = torch.randn(16 * rows + k, generator=gen(1)).cuda()
        given = flat.as_strided((rows, k), (16, 1))
        w = given.contiguous()
    elif kind == "columns one after the other":
        given = w.T.contiguous().T
    elif kind == "rows off the grid of 16 bytes":
        given = shifted(w, 1)
    else:
        given = w
    got_enc = enc
    if kind == "bytes off the grid":
        got_enc = Encoded(shifted(enc.codes, 1), shifted(enc.params, 1), shifted(enc.consts, 1), enc.sse)
    elif kind == "constants with spare columns":
        got_enc = Encoded(enc.codes, enc.params, torch.cat([enc.consts, enc.consts], 1), enc.sse)
    want = refine_groups([(w, enc, 4, 32)], hs, 2)[0]
    assert int((want != enc.codes).sum()) > 0
    assert torch.equal(refine_groups([(given, got_enc, 4, 32)], hs, 2)[0], want)


@pytest.mark.parametrize("k", [192, 640])
def test_highest_codes_as_a_column(k):
    from hi2_b200.refine import _decoded, _expand, refine_expanded

    w, enc, hs = encoded(40, k)
    lo_x, st_x = _expand(*_decoded(enc), 32)
    top = torch.full((40,), 15.0, device="cuda")
    want = refine_expanded(w, enc.codes, lo_x, st_x, top, hs, 2)
    assert torch.equal(refine_expanded(w, enc.codes, lo_x, st_x, top[:, None], hs, 2), want)


@pytest.mark.parametrize("k", [192, 640])
@pytest.mark.parametrize("form", ["groups", "expanded"])
def test_errors_are_freed_before_the_sweeps(form, k, monkeypatch):
    """The rows' errors (8 bytes a weight as TF32 parts) are read once, by the first product."""
    from hi2_b200 import refine, refine_kernel

    w, enc, hs = encoded(40, k)
    seen, sweeps = [], []
    name = "gemm_tc" if k >= refine.TC_MIN_K else "gemm"
    product, sweep = getattr(refine_kernel, name), refine_kernel.sweep

    def watch(a, *args, **kw):
        seen.append(weakref.ref(a))
        return product(a, *args, **kw)

    def check(*args):
        sweeps.append(seen[0]() is None)
        return sweep(*args)

    monkeypatch.setattr(refine_kernel, name, watch)
    monkeypatch.setattr(refine_kernel, "sweep", check)
    if form == "groups":
        refine.refine_groups([(w, enc, 4, 32)], hs, 2)
    else:
        lo_x, st_x = refine._expand(*refine._decoded(enc), 32)
        refine.refine_expanded(w, enc.codes, lo_x, st_x, torch.full((40,), 15.0, device="cuda"), hs, 2)
    assert sweeps and all(sweeps)
