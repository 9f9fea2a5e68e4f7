"""The error table in one search and one row pass against one candidate at a time: equal bits, over ragged
rows, rows and blocks of zeros, ladders whose step has no usable reciprocal, grouped column weights,
and candidate lists longer than a pass and longer than a call."""

import pytest
import torch

from helpers import gen, weights

pytestmark = pytest.mark.gpu

SIX = [(nb, b) for nb in (2, 4) for b in (16, 32, 64)]


def one_by_one(w, d, candidates, effort, row_group):
    from hi2_b200.encode import encode_rows

    encs = [encode_rows(w, d, nb, b, effort, want_codes=False, want_energy=True, row_group=row_group) for nb, b in candidates]
    return torch.stack([e.sse for e in encs]), encs[0].energy


@pytest.mark.parametrize("rows,k", [(1, 64), (3, 192), (33, 576), (70, 4160), (300, 1088)])
@pytest.mark.parametrize("kind", ["plain", "zeros", "tiny", "offset"])
@pytest.mark.parametrize("candidates", [SIX, SIX + [(8, 32), (8, 64)], [(8, 64), (1, 16), (3, 32)], SIX * 3])
def test_table_is_the_candidates_one_by_one(rows, k, kind, candidates):
    from hi2_b200.encode import EFFORT
    from hi2_b200.ladder_kernel import error_table

    w = weights(rows, k, rows + k)
    if kind == "zeros":
        w[:, : k // 2] = 0
        w[::3] = 0
    elif kind == "tiny":
        w = w * 1e-19  # steps round to fp16 zero
    elif kind == "offset":
        w = w + 40
    w = w.cuda()
    for groups in (1, 3):
        d = 0.05 + torch.rand(groups, k, generator=gen(k)).cuda()
        d = d[0].contiguous() if groups == 1 else d
        group = None if groups == 1 else torch.randint(0, groups, (rows,), generator=gen(rows)).cuda()
        for effort in ("fast", "normal"):
            sse, energy = error_table(w, d, candidates, EFFORT[effort]["grid"], EFFORT[effort]["ls"], group)
            want = one_by_one(w, d, candidates, effort, group)
            assert torch.equal(sse, want[0]) and torch.equal(energy, want[1])


def test_table_refuses_what_one_candidate_refuses():
    from hi2_b200.ladder_kernel import error_table

    w, d = torch.zeros(4, 96, device="cuda"), torch.ones(96, device="cuda")
    for bad in ([(2, 64)], [(2, 48)], [(9, 32)], [(0, 32)]):
        with pytest.raises(ValueError):
            error_table(w, d, bad, (0.0, 0.1), 1)
    with pytest.raises(RuntimeError):
        error_table(w, d, [], (0.0, 0.1), 1)


def test_threads_with_tables_of_different_widths():
    """Every call needs its own amount of shared memory; what a narrow table in one thread asks for does
    not take it from a wide one in another.  The entry point is called directly: the fewer of the
    interpreter's steps lie between two calls, the more often they meet."""
    import threading

    from hi2_b200 import _lib

    entry, failures = _lib.load().hi2_error_table, []
    nbits, blocks = _lib.host_i32([nb for nb, _ in SIX]), _lib.host_i32([b for _, b in SIX])

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            w, d, ladders, sse = torch.randn(1, k).cuda(), torch.ones(k).cuda(), torch.empty(2, k).cuda(), torch.empty(6).cuda()
            args = (_lib.ptr(w), k, _lib.ptr(d), None, _lib.host_floats((0.0,)), 1, 0, 6, nbits, blocks, 1, k, _lib.ptr(ladders[0]),
                    _lib.ptr(ladders[1]), _lib.ptr(sse), None, _lib.stream(w.device))
            for i in range(20000):
                if entry(*args):
                    failures.append((k, i, _lib.last_error()))
                if i % 64 == 0:
                    stream.synchronize()
            stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in (11008, 64, 64, 64)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]
