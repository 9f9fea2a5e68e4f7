"""The work a user of this package has it do, as single calls with their inputs.

Every case is one pass through public entry points, over the range of sizes of the workloads of
``bench.py`` (a 7B-shaped decoder layer: hidden 4096, FFN 11008; OLMoE experts: hidden 2048, FFN 1024;
the 1024-row k/v projections under grouped-query attention):

* ``moment``  the second moment of a Linear's calibration activations (``HessianStats.update``);
* ``factor``  basis change and damped inverse factor of one input (``transform_sigma``,
  ``inverse_factor``);
* ``table``   the error table of one weight at every candidate (``build_table``);
* ``gptq``    error-compensated rounding of one weight's rows, one job per candidate the allocator
  gave rows to (``encode_jobs_gptq``);
* ``refine``  +-1 refinement sweeps after the rounding (``refine_encoded``);
* ``layer``   statistics, factors, tables and encode of a decoder layer, or of a layer of experts, for
  given picks (``layer.accumulate`` ... ``layer.encode``).

``exact`` restates each of them in 64 bits with plain torch.
"""

import math

import torch

from hi2_b200 import layer as L
from hi2_b200.calibrate import ALL_CANDIDATES, INT8_CANDIDATES, Config, build_table
from hi2_b200.encode import EFFORT, Encoded
from hi2_b200.hessian import GptqJob, HessianStats, encode_jobs_gptq, inverse_factor, transform_sigma
from hi2_b200.refine import refine_encoded
from hi2_b200.stats import ColumnStats

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
F32, F64 = torch.float32, torch.float64
DAMP = 0.01

# rows per candidate that an allocation leaves: shares of (nbits, block)
MIXES = {
    "2.5bpw": (((2, 16), 0.15), ((2, 32), 0.30), ((2, 64), 0.35), ((4, 64), 0.20)),  # config 2, 5
    "3.0bpw": (((2, 16), 0.30), ((2, 32), 0.20), ((2, 64), 0.05), ((4, 32), 0.15), ((4, 64), 0.30)),  # config 1, 3
    "int8": (((2, 32), 0.55), ((4, 64), 0.44), ((8, 64), 0.01)),  # config 4: INT8 for the most sensitive rows
}


def listed():
    return [
        # an OLMoE expert with few routed tokens (8457 is the smallest count of that workload)
        {"name": "moment-expert", "kind": "moment", "k": 2048, "tokens": 8457, "dtype": "bf16"},
        # the widest input of a 7B-shaped layer, a 65536-token part of its calibration set
        {"name": "moment-ffn", "kind": "moment", "k": 11008, "tokens": 65536, "dtype": "bf16"},
        # the factors of an expert's down projection, of a hidden-sized input, of the FFN's
        {"name": "factor-expert", "kind": "factor", "k": 1024, "tokens": 8457},
        {"name": "factor-hidden", "kind": "factor", "k": 4096, "tokens": 16384},
        {"name": "factor-ffn", "kind": "factor", "k": 11008, "tokens": 22016},
        # tables: an expert's gate projection; a gate / up projection; k / v rows with INT8 open
        {"name": "table-expert", "kind": "table", "rows": 1024, "k": 2048, "dtype": "bf16", "effort": "normal", "int8": False},
        {"name": "table-ffn", "kind": "table", "rows": 11008, "k": 4096, "dtype": "bf16", "effort": "normal", "int8": False},
        # column loops: an attention projection at 3.0 bpw; the down projection at 2.5 bpw
        {"name": "gptq-hidden", "kind": "gptq", "rows": 4096, "k": 4096, "mix": "3.0bpw", "act_order": False},
        {"name": "gptq-ffn", "kind": "gptq", "rows": 4096, "k": 11008, "mix": "2.5bpw", "act_order": False},
        # the reference's default of two sweeps on an attention projection
        {"name": "refine-hidden", "kind": "refine", "rows": 4096, "k": 4096, "nbits": 2, "block": 32, "passes": 2},
        # whole calls: some experts of a layer, with uneven token counts; a 7B-shaped decoder layer
        {"name": "layer-experts", "kind": "layer", "experts": 5, "hidden": 2048, "ffn": 1024, "tokens": 8457, "mix": "2.5bpw"},
        {"name": "layer-llama", "kind": "layer", "experts": 0, "hidden": 4096, "ffn": 11008, "tokens": 32768, "mix": "3.0bpw"},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` between ``lo`` and ``hi``, spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["moment", "factor", "table", "table", "gptq", "gptq", "refine", "layer"])
    if kind == "moment":
        k = _log(rng, 1024, 11008, 16)
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        return {"kind": kind, "k": k, "tokens": _log(rng, 300, 16384 if dtype == "fp32" else 65536), "dtype": dtype}
    if kind == "factor":
        k = _log(rng, 512, 11008, 16)
        return {"kind": kind, "k": k, "tokens": 2 * k + rng.randrange(2 * k)}
    if kind == "table":
        return {"kind": kind, "rows": _log(rng, 129, 11008), "k": _log(rng, 1024, 4096, 64),
                "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"]), "effort": rng.choice(["fast", "normal", "normal", "max"]),
                "int8": rng.random() < 0.3}
    if kind == "gptq":
        return {"kind": kind, "rows": _log(rng, 129, 4096), "k": _log(rng, 1024, 11008, 64), "mix": rng.choice(sorted(MIXES)),
                "act_order": rng.random() < 0.2}
    if kind == "refine":
        nbits, block = rng.choice(ALL_CANDIDATES)
        return {"kind": kind, "rows": _log(rng, 129, 4096), "k": _log(rng, 1024, 4096, 64), "nbits": nbits, "block": block,
                "passes": rng.choice([1, 2, 2])}
    if rng.random() < 0.5:
        return {"kind": kind, "experts": rng.randrange(2, 6), "hidden": _log(rng, 1024, 2048, 64), "ffn": _log(rng, 512, 1024, 64),
                "tokens": _log(rng, 4096, 8457), "mix": rng.choice(["2.5bpw", "3.0bpw"])}
    return {"kind": kind, "experts": 0, "hidden": _log(rng, 1024, 4096, 64), "ffn": _log(rng, 2048, 11008, 64),
            "tokens": _log(rng, 24576, 32768), "mix": rng.choice(["2.5bpw", "3.0bpw"])}


# ---- inputs ------------------------------------------------------------------------------------
def _gen(seed, part=0):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * seed + part)


def _activations(tokens, k, seed, part, dtype):
    """N(0, 1) times a per-channel lognormal scale, with some correlation between neighbours."""
    g = _gen(seed, part)
    scale = torch.exp(torch.randn(1, k, generator=g, device=DEV))
    x = torch.empty(tokens, k, dtype=dtype, device=DEV)
    for t0 in range(0, tokens, 16384):
        n = min(16384, tokens - t0)
        z = torch.randn(n, k, generator=g, device=DEV)
        z[:, 1:] += 0.3 * z[:, :-1]
        x[t0 : t0 + n] = (z * scale).to(dtype)
    return x


def _weights(rows, k, seed, part, dtype):
    """N(0, 0.02) with rows of different sizes and 0.1 % of the input columns scaled up."""
    g = _gen(seed, part)
    w = 0.02 * torch.randn(rows, k, generator=g, device=DEV) * torch.exp(0.3 * torch.randn(rows, 1, generator=g, device=DEV))
    w[:, torch.randperm(k, generator=g, device=DEV)[: max(1, k // 1000)]] *= 8
    return w.to(dtype)


def _second_moment(x, out=F64):
    s = torch.zeros(x.shape[1], x.shape[1], dtype=F64, device=DEV)
    for t0 in range(0, x.shape[0], 16384):
        p = x[t0 : t0 + 16384].to(F64)
        s.addmm_(p.T, p)
    return s.to(out)


def _smoothing(diag):
    d = diag.to(F32).clamp_min(1e-12)
    return (d / d.log().mean().exp()).pow(0.25).clamp(0.05, 20.0).to(torch.float16)


def _hadamard():
    h = torch.ones(1, 1, dtype=F64, device=DEV)
    while h.shape[0] < 16:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)])
    return h / 4


def _rotated(x):
    """Every run of 16 columns of ``x`` multiplied by the order-16 Hadamard matrix."""
    return (x.to(F64).reshape(-1, x.shape[-1] // 16, 16) @ _hadamard()).reshape(x.shape)


def _stored_basis(sigma, s16):
    h = sigma.to(F64) / s16.to(F64) / s16.to(F64).reshape(-1, 1)
    return _rotated(_rotated(h).T.contiguous()).T.contiguous()


def _inverse_factor(hs):
    """Upper ``U`` with ``U^T U = (Hs + damp * mean(diag))^-1``, by one factorisation of the reversed matrix."""
    a = hs.to(F64).flip(0, 1).contiguous()
    a.diagonal().add_(DAMP * a.diagonal().mean())
    low = torch.linalg.cholesky(a)
    eye = torch.eye(a.shape[0], dtype=F64, device=DEV)
    return torch.linalg.solve_triangular(low, eye, upper=False).flip(0, 1).contiguous()


def _input(k, tokens, seed):
    """``(second moment [K, K] fp32, smoothing vector)`` of one calibrated input."""
    sigma = _second_moment(_activations(tokens, k, seed, 1, torch.bfloat16), F32)
    return sigma, _smoothing(sigma.diagonal() / tokens)


def _flags(k):
    return torch.ones(k // 16, dtype=torch.uint8)


def _stored_weights(case, s16, seed):
    w = _weights(case["rows"], case["k"], seed, 2, torch.bfloat16)
    return _rotated(w.to(F32) * s16.to(F32)).to(F32)


def _groups(rows, mix):
    """``[(nbits, block, number of rows)]`` of a mix, every row in one of them."""
    out, left = [], rows
    for i, ((nbits, block), share) in enumerate(MIXES[mix]):
        n = left if i + 1 == len(MIXES[mix]) else min(left, int(share * rows))
        left -= n
        if n:
            out.append((nbits, block, n))
    return out


def _candidates(case):
    return list(ALL_CANDIDATES) + (list(INT8_CANDIDATES) if case["int8"] else [])


# ---- the format's arithmetic in plain torch --------------------------------------------------------
def _round_div(a, b):
    return torch.round(a / torch.where(b == 0, torch.ones_like(b), b))


def _search(wb, db, n, effort):
    """Grid and least-squares search of ``(lo, step)`` per block, ``wb [N, nb, B]``, ``db [1, nb, B]``."""
    def err(lo, step):
        q = _round_div(wb - lo[..., None], step[..., None]).clamp_(0, n - 1)
        return (db * (lo[..., None] + q * step[..., None] - wb) ** 2).sum(-1), q

    mn, mx = wb.amin(-1), wb.amax(-1)
    span, best = mx - mn, None
    for a in EFFORT[effort]["grid"]:
        for b in EFFORT[effort]["grid"]:
            lo = mn + a * span
            step = (mx - b * span - lo) / (n - 1)
            e = err(lo, step)[0]
            if best is None:
                best = [lo, step, e]
            else:
                better = e < best[2]
                best = [torch.where(better, p, q) for p, q in zip((lo, step, e), best)]
    for _ in range(EFFORT[effort]["ls"]):
        q = err(best[0], best[1])[1]
        sd, sc, scc = db.sum(-1), (db * q).sum(-1), (db * q * q).sum(-1)
        sw, scw = (db * wb).sum(-1), (db * q * wb).sum(-1)
        det = sd * scc - sc * sc
        ok = det.abs() > 1e-20
        step = torch.where(ok, (sd * scw - sc * sw) / torch.where(ok, det, torch.ones_like(det)), torch.zeros_like(det))
        lo = torch.where(ok, (sw - step * sc) / sd.clamp_min(1e-20), wb.mean(-1))
        e = err(lo, step)[0]
        better = (e < best[2]) & (step > 0)
        best = [torch.where(better, p, q) for p, q in zip((lo, step, e), best)]
    return best[0], best[1]


def _bytes(lo, step):
    """``(params uint8 [N, nb, 2], consts fp16 [N, 3])`` of real ladders."""
    half = torch.float16
    step = step.clamp_min(0)
    ss = (step.amax(-1, keepdim=True) / 255).to(half)
    lm = lo.amin(-1, keepdim=True).to(half)
    ls = ((lo.amax(-1, keepdim=True) - lm.to(lo.dtype)).clamp_min(0) / 255).to(half)
    su = _round_div(step, ss.to(lo.dtype)).clamp(0, 255) * (ss > 0)
    lu = _round_div(lo - lm.to(lo.dtype), ls.to(lo.dtype)).clamp(0, 255) * (ls > 0)
    return torch.stack([lu, su], -1).to(torch.uint8), torch.cat([lm, ls, ss], -1)


def _decoded(params, consts, dtype):
    c = consts.to(F64)
    lo = (params[..., 0].to(F64) * c[:, 1:2] + c[:, 0:1]).to(torch.float16)
    step = (params[..., 1].to(F64) * c[:, 2:3]).to(torch.float16)
    return lo.to(dtype), step.to(dtype)


def _ladders(w, d, nbits, block, effort):
    """Searched and quantised ladders of the rows ``w`` in the precision of ``w``, in runs of rows."""
    k, parts = w.shape[1], []
    per = max(1, (1 << 24) // k)
    for r0 in range(0, w.shape[0], per):
        wb = w[r0 : r0 + per].reshape(-1, k // block, block)
        parts.append(_bytes(*_search(wb, d.to(w.dtype).reshape(1, -1, block), 2**nbits, effort)))
    return torch.cat([p for p, _ in parts]), torch.cat([c for _, c in parts])


def _value(lo, q, step):
    return (lo + q * step).to(torch.float16).to(lo.dtype)


def _error(w, d, codes, lo, step, block):
    rec = _value(lo.repeat_interleave(block, 1), codes, step.repeat_interleave(block, 1))
    return (d.to(w.dtype) * (rec - w) ** 2).sum(-1)


def _round_columns(w, u, lo, step, nbits, block, order):
    """Codes ``[N, K]`` of the error-compensated column loop, in the precision of ``w``."""
    work, codes = w[:, order].clone(), torch.empty_like(w)
    at = order.tolist()
    for c0 in range(0, len(at), 128):
        c1 = min(c0 + 128, len(at))
        seg, errs = work[:, c0:c1].clone(), torch.empty_like(work[:, c0:c1])
        tri = u[c0:c1, c0:c1]
        for i in range(c1 - c0):
            b = at[c0 + i] // block
            q = _round_div(seg[:, i] - lo[:, b], step[:, b]).clamp_(0, 2**nbits - 1)
            q = torch.where(step[:, b] == 0, torch.zeros_like(q), q)
            e = (seg[:, i] - _value(lo[:, b], q, step[:, b])) / tri[i, i]
            seg.addr_(e, tri[i], alpha=-1)
            errs[:, i], codes[:, at[c0 + i]] = e, q
        work[:, c1:] -= errs @ u[c0:c1, c1:]
    return codes


def _sweeps(w, codes, lo, step, hs, nbits, block, passes):
    """Codes after +-1 refinement sweeps, in the precision of ``w``."""
    lo, step, c = lo.repeat_interleave(block, 1), step.repeat_interleave(block, 1), codes.to(w.dtype)
    g = (_value(lo, c, step) - w) @ hs
    hd = hs.diagonal()
    for _ in range(passes):
        for c0 in range(0, w.shape[1], 128):
            c1 = min(c0 + 128, w.shape[1])
            seg, moved, hb = g[:, c0:c1].clone(), torch.empty_like(w[:, c0:c1]), hs[c0:c1, c0:c1]
            now = _value(lo[:, c0:c1], c[:, c0:c1], step[:, c0:c1])
            change, can = [], []
            for sign in (1.0, -1.0):
                q = c[:, c0:c1] + sign
                change.append(_value(lo[:, c0:c1], q, step[:, c0:c1]) - now)
                can.append((q >= 0) & (q <= 2**nbits - 1) & (step[:, c0:c1] > 0))
            change, can = torch.stack(change), torch.stack(can)
            for i in range(c1 - c0):
                dw = change[:, :, i]
                gain = torch.where(can[:, :, i], -(2 * dw * seg[:, i] + dw * dw * hd[c0 + i]), -torch.inf)
                best, which = gain.max(0)
                move = torch.where(best > 0, dw.gather(0, which[None])[0], 0.0)
                c[:, c0 + i] += torch.where(best > 0, 1.0 - 2.0 * which, 0.0)
                moved[:, i] = move
                seg.addr_(move, hb[i])
            g += moved @ hs[c0:c1]
    return c


def _refine_start(case, seed):
    """Stored rows, their rounding after the column loop, and the Hessian, all in 32 bits."""
    sigma, s16 = _input(case["k"], 4 * case["k"], seed)
    hs = _stored_basis(sigma / (4 * case["k"]), s16)
    hs = ((hs + hs.T) / 2).to(F32)
    w, d = _stored_weights(case, s16, seed), hs.diagonal()
    params, consts = _ladders(w, d, case["nbits"], case["block"], "fast")
    lo, step = _decoded(params, consts, F32)
    order = torch.arange(case["k"], device=DEV)
    codes = _round_columns(w, _inverse_factor(hs).to(F32), lo, step, case["nbits"], case["block"], order)
    return w, hs, codes.to(torch.uint8), params, consts


def _gptq_start(case, seed):
    """Stored rows, ladder weights, factor and column order of one tensor."""
    sigma, s16 = _input(case["k"], 2 * case["k"], seed)
    hs = _stored_basis(sigma / (2 * case["k"]), s16)
    d = hs.diagonal().to(F32)
    perm = torch.argsort(d, descending=True) if case["act_order"] else None
    if perm is not None:
        hs = hs[perm][:, perm]
    return _stored_weights(case, s16, seed), d, _inverse_factor(hs).to(F32), perm


def _layer_parts(case, seed):
    if case["experts"]:
        h, f = case["hidden"], case["ffn"]
        shapes, widths, reads, tokens = {}, {}, {}, {}
        for e in range(case["experts"]):
            for p, shape, x in (("gate_proj", (f, h), "in"), ("up_proj", (f, h), "in"), ("down_proj", (h, f), "mid")):
                shapes[f"experts.{e}.{p}"], reads[f"experts.{e}.{p}"] = shape, f"experts.{e}.{x}"
            widths[f"experts.{e}.in"], widths[f"experts.{e}.mid"] = h, f
            tokens[f"experts.{e}.in"] = tokens[f"experts.{e}.mid"] = case["tokens"] + 997 * e
        plan = L.LayerPlan(reads)
    else:
        shapes, widths = L.llama_shapes(case["hidden"], case["ffn"])
        plan, tokens = L.llama_plan(), {n: case["tokens"] for n in widths}
    return shapes, widths, plan, tokens


def prepare(case, seed):
    kind = case["kind"]
    if kind == "moment":
        return {"case": case, "x": _activations(case["tokens"], case["k"], seed, 1, DTYPES[case["dtype"]])}
    if kind == "factor":
        sigma, s16 = _input(case["k"], case["tokens"], seed)
        return {"case": case, "sigma": sigma, "s16": s16, "flags": _flags(case["k"])}
    if kind == "table":
        k = case["k"]
        x = _activations(4096, k, seed, 1, torch.bfloat16).to(F64).reshape(4096, k // 16, 16).transpose(0, 1)
        stats = ColumnStats.from_state({"S": x.transpose(1, 2) @ x, "n": 4096, "k": k}, DEV)
        s16 = _smoothing(stats.S.diagonal(dim1=1, dim2=2).flatten() / 4096)
        cfg = Config(candidates=_candidates(case), effort=case["effort"])
        return {"case": case, "w": _weights(case["rows"], k, seed, 2, DTYPES[case["dtype"]]), "stats": stats, "cfg": cfg,
                "transform": (s16, _flags(k))}
    if kind == "gptq":
        w, d, u, perm = _gptq_start(case, seed)
        jobs, r0 = [], 0
        for nbits, block, n in _groups(case["rows"], case["mix"]):
            jobs.append(GptqJob(w[r0 : r0 + n], d, u, nbits, block, perm))
            r0 += n
        return {"case": case, "jobs": jobs}
    if kind == "refine":
        w, hs, codes, params, consts = _refine_start(case, seed)
        return {"case": case, "w": w, "hs": hs, "enc": Encoded(codes, params, consts, torch.zeros(case["rows"], device=DEV))}
    shapes, widths, plan, tokens = _layer_parts(case, seed)
    cfg = Config()
    at = {c: i for i, c in enumerate(cfg.candidates)}
    weights, picks = {}, {}
    for i, (name, (r, k)) in enumerate(shapes.items()):
        weights[name] = _weights(r, k, seed, 100 + i, torch.bfloat16)
        mine = torch.cat([torch.full((n,), at[nbits, block]) for nbits, block, n in _groups(r, case["mix"])])
        picks[name] = mine[torch.randperm(r, generator=torch.Generator().manual_seed(seed + i))]
    inputs = {n: _activations(tokens[n], k, seed, 200 + i, torch.bfloat16) for i, (n, k) in enumerate(widths.items())}
    return {"case": case, "weights": weights, "picks": picks, "inputs": inputs, "plan": plan, "cfg": cfg}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "moment":
        h = HessianStats(case["k"], DEV)
        h.update(state["x"])
        return {"S": h.S}
    if kind == "factor":
        hs, d = transform_sigma(state["sigma"], state["s16"], state["flags"], denom=float(case["tokens"]), return_diag=True)
        return {"hs": hs, "d": d, "u": inverse_factor(hs, DAMP)}
    if kind == "table":
        t = build_table("w", state["w"], state["stats"], state["cfg"], transform=state["transform"])
        return {"sse": t.sse, "energy": t.energy}
    if kind == "gptq":
        encs = encode_jobs_gptq(state["jobs"])
        return [{"codes": e.codes, "params": e.params, "consts": e.consts, "sse": e.sse} for e in encs]
    if kind == "refine":
        e = refine_encoded(state["enc"], state["w"], state["hs"], case["nbits"], case["block"], case["passes"])
        return {"codes": e.codes, "sse": e.sse}
    cfg, weights, plan = state["cfg"], state["weights"], state["plan"]
    shared = L.accumulate(state["inputs"], DEV, defer_check=True)
    L.finish_statistics(shared, cfg)
    factors = L.start_factors(shared, cfg, DEV)
    tables = L.tabulate(weights, plan, shared, cfg, grouped=bool(case["experts"]))
    packed = L.encode(weights, plan, shared, tables, state["picks"], cfg, factors=factors)
    # the code stream as bytes: a code that falls on the other side of a tie changes one of them
    return {n: {"sse": tables[n].sse, "codes": t.codes.view(torch.uint8), "params": t.blk_params, "consts": t.row_consts}
            for n, t in packed.items()}


def work(case):
    kind = case["kind"]
    if kind == "moment":
        k, t = case["k"], case["tokens"]
        return {"bytes": t * k * (4 if case["dtype"] == "fp32" else 2) + 4 * k * k, "flops": t * k * (k + 1)}
    if kind == "factor":  # two triangular halves: factorisation and inverse
        return {"bytes": 12 * case["k"] ** 2, "flops": 2 * case["k"] ** 3 // 3}
    if kind == "table":
        e, c, n = EFFORT[case["effort"]], len(_candidates(case)), case["rows"] * case["k"]
        return {"bytes": n * (4 if case["dtype"] == "fp32" else 2) + 4 * c * case["rows"],
                "flops": n * c * (8 * len(e["grid"]) ** 2 + 20 * e["ls"])}
    if kind == "gptq":  # one ladder search and a triangular product per row
        r, k = case["rows"], case["k"]
        return {"bytes": r * k * 5 + 2 * k * k, "flops": r * k * k + r * k * (8 * 36 + 20 * 2)}
    if kind == "refine":  # g = e Hs, and every sweep's moves through Hs
        r, k = case["rows"], case["k"]
        return {"bytes": r * k * 6 + 4 * k * k, "flops": 2 * r * k * k * (1 + case["passes"])}
    shapes, widths, _, tokens = _layer_parts(case, 0)
    b = f = 0
    for n, k in widths.items():
        b, f = b + 2 * tokens[n] * k, f + tokens[n] * k * (k + 1) + 2 * k**3 // 3
    for r, k in shapes.values():
        b, f = b + 2 * r * k + r * k * 3 // 8, f + r * k * k + 7 * r * k * (8 * 36 + 20 * 2)
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times the distance to ``exact`` (or, where codes come back, to a 64-bit column loop
    over the same ladders), measured over the listed and eight drawn cases."""
    kind = case["kind"]
    if kind == "moment":  # fp32 sums of exact products in tensor memory: 2.2e-6
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "factor":  # an fp32-grade factorisation of a damped Hessian: 1.2e-6, 2.1e-4
        return {"rel": 5e-6, "max": 1e-3}
    if kind == "table":  # fp32 sums; a ladder on the other side of a tie moves one row: 5e-6, 2.4e-4
        return {"rel": 2e-5, "max": 1e-3}
    # A code within the rounding error of the trailing update of a tie goes the other way and the rest
    # of its row follows it; ladders do not depend on it.
    if kind == "gptq":  # 4.6e-4 of the codes, and 1e-3 (one row: 2.3e-2) of the errors that follow from them
        return {"rel": 4e-3, "max": 0.1, "differ": 2e-3}
    if kind == "refine":  # 1.1e-5 of the codes, 1.8e-4 (one row: 7.5e-3) of the errors
        return {"rel": 7e-4, "max": 3e-2, "differ": 1e-4}
    # tables as above through the inputs' own moments; up to four codes share a byte of the stream
    return {"rel": 2e-5, "max": 1e-3, "differ": 8e-3}


def exact(case, seed):
    kind = case["kind"]
    if kind == "moment":
        return {"S": _second_moment(_activations(case["tokens"], case["k"], seed, 1, DTYPES[case["dtype"]]))}
    if kind == "factor":
        sigma, s16 = _input(case["k"], case["tokens"], seed)
        hs = _stored_basis(sigma.to(F64) / case["tokens"], s16)
        return {"hs": hs, "d": hs.diagonal().clone(), "u": _inverse_factor(hs)}
    if kind == "table":
        st = prepare(case, seed)
        s16 = st["transform"][0].to(F64)
        w = _rotated(st["w"].to(F64) * s16)
        m = st["stats"].S / 4096 / s16.reshape(-1, 16, 1) / s16.reshape(-1, 1, 16)
        d = (_hadamard() @ m @ _hadamard()).diagonal(dim1=1, dim2=2).flatten()
        sse = []
        for nbits, block in _candidates(case):
            lo, step = _decoded(*_ladders(w, d, nbits, block, case["effort"]), F64)
            codes = _round_div(w - lo.repeat_interleave(block, 1), step.repeat_interleave(block, 1)).clamp_(0, 2**nbits - 1)
            codes = codes * (step > 0).repeat_interleave(block, 1)
            sse.append(_error(w, d, codes, lo, step, block))
        return {"sse": torch.stack(sse), "energy": (d * w**2).sum()}
    if kind == "gptq":
        w, d, u, perm = _gptq_start(case, seed)
        w, u, out, r0 = w.to(F64), u.to(F64), [], 0
        order = torch.arange(case["k"], device=DEV) if perm is None else perm
        for nbits, block, n in _groups(case["rows"], case["mix"]):
            rows = w[r0 : r0 + n]
            lo, step = _decoded(*_ladders(rows, d, nbits, block, "normal"), F64)
            codes = _round_columns(rows, u, lo, step, nbits, block, order)
            out.append({"codes": None, "params": None, "consts": None, "sse": _error(rows, d, codes, lo, step, block)})
            r0 += n
        return out
    if kind == "refine":
        w, hs, codes, params, consts = _refine_start(case, seed)
        w, hs = w.to(F64), hs.to(F64)
        lo, step = _decoded(params, consts, F64)
        codes = _sweeps(w, codes, lo, step, hs, case["nbits"], case["block"], case["passes"])
        return {"codes": None, "sse": _error(w, hs.diagonal(), codes, lo, step, case["block"])}
    return None  # a whole layer in 64 bits takes longer than its parts, which the other cases hold
