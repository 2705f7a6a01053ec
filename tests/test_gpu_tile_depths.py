"""Tiles chosen from a batch's sizes hold instances whose live points are many
for their items: a small item among large ones, and containers that the items
leave open. No restart outgrows its tile, solved or served."""
import os
import random
import re
import subprocess
import sys

import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _cartons(n, lo, hi, extra, seed):
    """n cartons, each a type of its own, and one cube of edge `extra` (0: none)."""
    rng = random.Random(seed)
    types = [tuple(rng.randint(lo, hi) for _ in range(3)) for _ in range(n)]
    types += [(extra,) * 3] if extra else []
    rows = "".join(f"{i} {a} 1 {b} 1 {c} 1 1\n" for i, (a, b, c) in enumerate(types, 1))
    return f"1\n1 {seed}\n587 233 220\n{len(types)}\n{rows}"


def _with_cube(text, edge):
    lines = text.rstrip().splitlines()
    n = int(lines[3]) + 1
    return "\n".join(lines[:3] + [str(n)] + lines[4:] + [f"{n} {edge} 1 {edge} 1 {edge} 1 1"]) + "\n"


def _texts(family):
    if family == "cube_2cm":
        return [_with_cube(synth.batched(30000 + i).to_thpack(), 2) for i in range(6)]
    if family == "cartons_and_4cm":
        return [_cartons(120, 30, 80, 4, i) for i in range(6)]
    return [_cartons(250, 20, 60, 0, i) for i in range(6)]


FAMILIES = ["cube_2cm", "cartons_and_4cm", "open_250"]


def _check(texts, res, restarts):
    for t, r in list(zip(texts, res))[::3]:
        oi = O.OInstance(t)
        for k in range(0, restarts, max(1, restarts // 3)):
            assert O.strip_time(r.json(k)) == O.strip_time(O.run(oi, seed=k)[0]), k


@pytest.mark.parametrize("n,restarts,launches", [(1, 64, 2), (6, 64, 2), (6, 1024, 4)])
@pytest.mark.parametrize("family", FAMILIES)
def test_no_restart_runs_again_on_the_host(family, n, restarts, launches):
    """One wave: decoder and selection. Several: with the retry stage's two."""
    texts = _texts(family)[:n]
    with P.Handle() as h:
        b = h.prepare([P.Instance.parse(t) for t in texts], P.make_opts(seed=0, restarts=restarts))
        assert b.run()[2] == launches
        _check(texts, b.fetch(), restarts)
        b.close()


@pytest.mark.parametrize("n,restarts,launches", [(1, 64, 2), (6, 512, 4)])
def test_block_engine_of_single_copies(n, restarts, launches):
    """Every carton is a type of its own, so a block is a box."""
    texts = _texts("open_250")[:n]
    kw = dict(amax=3, bmax=3, kmax=3, topk=16)
    with P.Handle() as h:
        b = h.prepare([P.Instance.parse(t) for t in texts],
                            P.make_opts(seed=0, restarts=restarts, eps=0.5, engine="block", **kw))
        assert b.run()[2] == launches
        r = b.fetch()[0]
        for k in (0, restarts - 1):
            want = O.run_block(O.OInstance(texts[0]), seed=k, eps=0.5, **kw)
            assert O.strip_time(r.json(k)) == O.strip_time(want), k
        b.close()


SERVED = """
import sys
sys.path[:0] = {paths!r}
import test_gpu_tile_depths as T
import plpb200 as P
plain = [T.synth.batched(30010 + i).to_thpack() for i in range(6)]
deep = T._texts("cube_2cm")[:2] + T._texts("cartons_and_4cm")[:2] + T._texts("open_250")[:2]
deep += ["1\\n1 9\\n587 233 220\\n1\\n1 20 1 20 1 20 1 300\\n"]
texts = {order}
with P.Handle() as h:
    ids = [h.submit(P.Instance.parse(t), P.make_opts(seed=0, restarts=192)) for t in texts]
    for rid in ids:
        assert h.wait(rid, 60000) == P.OK, P.last_error()
    T._check(texts, [h.take(rid) for rid in ids], 192)
    c = h.serve_counters()
assert c["served"] == len(texts) and c["fallbacks"] == 0, c
"""


@pytest.mark.parametrize("order", ["deep + plain", "plain + deep + plain"])
def test_served_requests_stay_with_the_main_decoders(order):
    """Also after a launch that started with others (it is drained for them)."""
    env = dict(os.environ, PLP_SERVE_TRACE="1")
    code = SERVED.format(paths=[os.path.join(os.path.dirname(HERE), "plp-gpu_b200"), HERE], order=order)
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env)
    assert p.returncode == 0, p.stderr[-2000:]
    ended = re.findall(r"launch ended head=\d+ overflow=(\d+)/(\d+)", p.stderr)
    assert ended and all(b == "0" for _, b in ended), ended
