"""The decoder drops points whose smallest-edge cuboid meets a box or the
container wall. Small containers with edges down to 1, one-axis orientation
sets (the smallest edge differs per axis), types that fit nowhere and types
of quantity zero, each restart against the CPU oracle (exact equality)."""
import random

import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu


def _instance(rng, lo, hi, flags):
    L, W, H = rng.randint(8, 40), rng.randint(8, 40), rng.randint(8, 40)
    n = rng.randint(1, 6)
    lines = ["1", "1 5", f"{L} {W} {H}", str(n)]
    for i in range(1, n + 1):
        e = [rng.randint(lo, hi) for _ in range(3)]
        if i == 1 and rng.random() < 0.3:
            e[0] = 50                      # longer than the container
        f = flags(rng)
        q = 0 if n > 1 and i == n and rng.random() < 0.3 else rng.randint(1, 25)
        lines.append(f"{i} {e[0]} {f[0]} {e[1]} {f[1]} {e[2]} {f[2]} {q}")
    return "\n".join(lines) + "\n"


FLAGS = {"all": lambda r: (1, 1, 1), "upright": lambda r: (0, 0, 1),
         "mixed": lambda r: r.choice([(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 1, 1)])}


@pytest.mark.parametrize("flags", sorted(FLAGS))
@pytest.mark.parametrize("lo,hi", [(1, 6), (2, 9), (4, 5), (3, 14)])
def test_dead_point_rule_matches_oracle(flags, lo, hi):
    rng = random.Random(lo * 100 + hi)
    texts = [_instance(rng, lo, hi, FLAGS[flags]) for _ in range(24)]
    insts = [P.Instance.parse(t) for t in texts]
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=4, eps=0.5, theta=0.6))
    for n, (t, r) in enumerate(zip(texts, res)):
        oi = O.OInstance(t)
        for k in range(4):
            js, _, _ = O.run(oi, seed=k, eps=0.5, theta=0.6)
            assert O.strip_time(r.json(k)) == O.strip_time(js), (n, k, t)


def test_dead_point_rule_on_the_stress_family():
    """Partial rotation flags at full size, every restart on the random branch."""
    texts = [synth.stress(42000 + i).to_thpack() for i in range(4)]
    insts = [P.Instance.parse(t) for t in texts]
    with P.Handle() as h:
        res = h.solve(insts, P.make_opts(seed=0, restarts=6, eps=1.0))
    for t, r in zip(texts, res):
        oi = O.OInstance(t)
        for k in range(6):
            js, _, _ = O.run(oi, seed=k, eps=1.0)
            assert O.strip_time(r.json(k)) == O.strip_time(js), k
