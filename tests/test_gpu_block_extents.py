"""Block engine on the decoder's points (free extents, dead points, marked
points): small containers with edges down to 1, one-axis orientation sets, deep
blocks and every pick rule, each restart against the CPU oracle."""
import random

import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu


def _instance(rng, lo, hi):
    L, W, H = rng.randint(8, 40), rng.randint(8, 40), rng.randint(8, 40)
    n = rng.randint(1, 5)
    lines = ["1", "1 5", f"{L} {W} {H}", str(n)]
    for i in range(1, n + 1):
        e = [rng.randint(lo, hi) for _ in range(3)]
        f = rng.choice([(1, 1, 1), (0, 0, 1), (1, 0, 0), (1, 1, 0)])
        lines.append(f"{i} {e[0]} {f[0]} {e[1]} {f[1]} {e[2]} {f[2]} {rng.randint(1, 30)}")
    return "\n".join(lines) + "\n"


@pytest.mark.parametrize("pick", ["first", "support", "contact"])
@pytest.mark.parametrize("lo,hi,amax", [(1, 5, 4), (2, 8, 3), (4, 5, 1)])
def test_block_points_match_oracle(pick, lo, hi, amax):
    rng = random.Random(lo * 10 + hi)
    texts = [_instance(rng, lo, hi) for _ in range(16)]
    insts = [P.Instance.parse(t) for t in texts]
    kw = dict(amax=amax, bmax=amax, kmax=amax, topk=16, eps=0.5, pick=pick, theta=0.6)
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=4, engine="block", **kw))
    for n, (t, r) in enumerate(zip(texts, res)):
        oi = O.OInstance(t)
        for k in range(4):
            assert O.strip_time(r.json(k)) == O.strip_time(O.run_block(oi, seed=k, **kw)), (n, k, t)


def test_block_campaign_batch_matches_oracle_samples():
    """Several waves, seeds shared by the instances (seeded states from the table)."""
    texts = [i.to_thpack() for i in synth.batched_set(48, 37000)]
    insts = [P.Instance.parse(t) for t in texts]
    kw = dict(amax=4, bmax=4, kmax=6, topk=64, eps=0.5, theta=0.9)
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=64, engine="block", **kw))
    for n, (t, r) in enumerate(zip(texts, res)):
        oi = O.OInstance(t)
        for k in range(n % 9, 64, 23):
            assert O.strip_time(r.json(k)) == O.strip_time(O.run_block(oi, seed=k, **kw)), (n, k)
