"""Multi-pass restarts of a batch of unequal instances: every resident decoder
keeps the pass it is running in a row of scratch of its own, so restarts of
instances with different item counts that run at the same time must not touch
each other's rows."""
import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu

OPTS = dict(eps=0.3, theta=0.5, order="input", mu=0.45)


@pytest.mark.parametrize("best_only", [False, True])
def test_multi_pass_batch_of_unequal_instances_matches_oracle(best_only):
    texts = [i.to_thpack() for i in synth.batched_set(24, 36000)] + [synth.single_pass(3).to_thpack()]
    insts = [P.Instance.parse(t) for t in texts]
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=32, passes=3, best_only=best_only, **OPTS))
    for n, (t, r) in enumerate(zip(texts, res)):
        oi = O.OInstance(t)
        for k in [r.best()[0]] if best_only else range(n % 5, 32, 9):
            js, _, _ = O.run(oi, seed=k, passes=3, **OPTS)
            assert O.strip_time(r.json(k)) == O.strip_time(js), (n, k)


def test_block_engine_multi_pass_batch_of_unequal_instances_matches_oracle():
    texts = [i.to_thpack() for i in synth.batched_set(16, 36100)]
    insts = [P.Instance.parse(t) for t in texts]
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=24, passes=3, eps=0.5, theta=0.5, engine="block"))
    for n, (t, r) in enumerate(zip(texts, res)):
        oi = O.OInstance(t)
        for k in range(n % 5, 24, 7):
            exp = O.run_block(oi, seed=k, passes=3, eps=0.5, theta=0.5)
            assert O.strip_time(r.json(k)) == O.strip_time(exp), (n, k)
