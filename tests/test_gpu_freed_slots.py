"""More points made dead by one placement than the placement notes slots (32):
the slots left over come back with the next placement, wherever its box lies."""
import pytest

import oracle_py as O
import plpb200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["ep", "block"])
@pytest.mark.parametrize("g,W,n,C,points", [(8, 150, 60, 96, 81), (10, 190, 90, 160, 126), (12, 230, 140, 224, 182)])
def test_slots_past_the_32nd_come_back(engine, g, W, n, C, points):
    """g x g cubes on the floor, a slab over all of them (g * g points dead at
    once), then cubes on the floor beside them, which reach past none of those:
    at most `points` live points (107, 194 and 294 slots with the dead ones kept)."""
    assert points <= C
    text = f"1\n1 1\n{10 * g} {W} 60\n3\n1 10 0 10 0 10 1 {g * g}\n2 {10 * g} 0 {10 * g} 0 5 1 1\n3 9 0 9 0 9 1 {n}\n"
    kw = dict(amax=1, bmax=1, kmax=1, topk=1) if engine == "block" else dict(order="input")
    opts = P.make_opts(seed=0, restarts=2, eps=0.0, theta=None, engine=engine, **kw)
    with P.Handle() as h:
        h.set_tile(288, C, 1, 1, 1)
        b = h.prepare([P.Instance.parse(text)], opts)
        launches = b.run()[2]
        r = b.fetch()[0]
        if engine == "block":
            kw.pop("order", None)
            want = O.run_block(O.OInstance(text), seed=1, eps=0.0, theta=None, **kw)
        else:
            want = O.run(O.OInstance(text), seed=1, eps=0.0, theta=None, order="input")[0]
        assert O.strip_time(r.json(1)) == O.strip_time(want)
        if engine == "ep":        # the block engine places by volume: no slab after the cubes
            assert launches == 2
        b.close()
