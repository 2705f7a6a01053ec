"""Served results read the pinned block that the decoders wrote: blocks given
back and taken again, results that outlive the handle, and more results held
than there are blocks for (those are copied)."""
import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu

PICK = (0, 1, 31, 512, 1023)


def _rows(r):
    return [O.strip_time(r.json(k)) for k in PICK]


def test_held_and_returned_blocks_keep_their_results():
    texts = [i.to_thpack() for i in synth.batched_set(4, 37400)]
    insts = [P.Instance.parse(t) for t in texts]
    opts = P.make_opts(seed=5, restarts=1024)
    h = P.Handle()
    solved = h.solve(insts, opts)
    want, best = [_rows(r) for r in solved], [r.best() for r in solved]
    for t, rows in zip(texts, want):
        oi = O.OInstance(t)
        for k, row in zip(PICK, rows):
            assert row == O.strip_time(O.run(oi, seed=5 + k)[0])
    held, total = [], 0
    for burst in range(6):
        n = 40
        ids = [h.submit(insts[q % 4], opts) for q in range(n)]
        for q, rid in enumerate(ids):
            assert h.wait(rid) == P.OK
            r = h.take(rid)
            if burst in (1, 3) and q % 3 == 0:      # given back at once, out of order with the others
                assert _rows(r) == want[q % 4]
                continue
            held.append((q % 4, r))
        total += n
    assert h.serve_counters()["served"] == total
    h.close()
    for i, r in held:
        assert r.best() == best[i]
        assert _rows(r) == want[i]
    del held, r
