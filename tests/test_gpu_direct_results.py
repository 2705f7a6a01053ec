"""Placements that the decoders write into the pinned result block themselves,
against the copied path (pool off), the automatic tile and the oracle: tiles
that restarts outgrow in one wave (host retries) and in several (the retry
stage on the device), and containers without a top-z index."""
import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu


def _jsons(res):
    return [[O.strip_time(r.json(k)) for k in range(r.restarts)] for r in res]


def _solve(insts, opts, tile=None):
    with P.Handle() as h:
        if tile:
            h.set_tile(*tile)
        return _jsons(h.solve(insts, opts))


@pytest.mark.parametrize("n,restarts", [(1, 1), (1, 33), (5, 40), (32, 160)])
@pytest.mark.parametrize("tile", [(32, 64, 1, 1, 16), (32, 128, 1, 4, 1)])
def test_outgrown_tiles_write_the_same_results(n, restarts, tile, monkeypatch):
    texts = [i.to_thpack() for i in synth.batched_set(n, 37300)]
    insts = [P.Instance.parse(t) for t in texts]
    opts = P.make_opts(seed=3, restarts=restarts)
    direct = _solve(insts, opts, tile)
    assert direct == _solve(insts, opts)          # the tile chosen from the sizes
    monkeypatch.setenv("PLP_PINNED_POOL_MB", "0")
    assert direct == _solve(insts, opts, tile)
    for t, rows in list(zip(texts, direct))[::5]:
        oi = O.OInstance(t)
        for k in range(0, restarts, 37):
            assert rows[k] == O.strip_time(O.run(oi, seed=3 + k)[0]), k


@pytest.mark.parametrize("engine", ["ep", "block"])
@pytest.mark.parametrize("H", [4090, 4095, 9000])
def test_no_top_z_index(engine, H):
    """4096 entries are the index's largest size; taller containers search the
    sorted tops instead."""
    text = f"1\n1 5\n60 50 {H}\n3\n1 30 0 25 0 700 1 30\n2 20 1 25 1 500 1 30\n3 17 1 13 1 11 1 40\n"
    kw = dict(amax=3, bmax=3, kmax=3, topk=16) if engine == "block" else {}
    with P.Handle() as h:
        (r,) = h.solve([P.Instance.parse(text)],
                       P.make_opts(seed=0, restarts=5, eps=0.5, theta=0.6, engine=engine, **kw))
    oi = O.OInstance(text)
    for k in range(5):
        want = (O.run_block(oi, seed=k, eps=0.5, theta=0.6, **kw) if engine == "block"
                else O.run(oi, seed=k, eps=0.5, theta=0.6)[0])
        assert O.strip_time(r.json(k)) == O.strip_time(want), k
