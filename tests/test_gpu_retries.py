"""Retries of restarts that outgrow a shallow hand-set tile: boxes and points
grow one at a time, as often as it takes."""
import pytest

import oracle_py as O
import plpb200 as P
from test_gpu_tile_depths import _cartons

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["ep", "block"])
@pytest.mark.parametrize("tile", [(16, 32, 1, 1, 1), (32, 32, 1, 1, 16)])
def test_shallow_tiles_grow_as_often_as_it_takes(engine, tile):
    """250 cartons, a type each: 250 boxes and some 300 points, four doublings
    of either from the shallower tile."""
    text = _cartons(250, 20, 60, 0, 1)
    kw = dict(amax=1, bmax=1, kmax=1, topk=4) if engine == "block" else {}
    with P.Handle() as h:
        h.set_tile(*tile)
        r = h.solve([P.Instance.parse(text)], P.make_opts(seed=3, restarts=2, engine=engine, **kw))[0]
    for k in range(2):
        oi = O.OInstance(text)
        want = O.run_block(oi, seed=3 + k, **kw) if engine == "block" else O.run(oi, seed=3 + k)[0]
        assert O.strip_time(r.json(k)) == O.strip_time(want)
