"""Cases that time the framework through its public entry points.

Each case is one call pattern of a program that uses the library: a lone solve,
a multi-restart solve, batches up to the largest one the library is built for,
a burst of served requests, the block-building engine, the one-step
feasibility call (on its own and inside the plain decode loop) and the
allocation-free decode into caller-owned device buffers. Instances are the
seeded synthetic ones of ``plpb200.synth`` (587 x 233 x 220 container).

A case is a dict of plain values: ``kind`` names the entry point, the other
keys are its sizes and options. ``prepare`` makes the instances, handle and
buffers a program has before the call; ``run`` is the call and the reading of
its answer; ``exact`` gives the same answer from a plain Python decoder where
that takes seconds.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "plp-gpu_b200"))

import plpb200 as P  # noqa: E402
from plpb200 import synth  # noqa: E402

L, W, H = synth.CONTAINER
_GEN = {"single_pass": synth.single_pass, "multi_restart": synth.multi_restart, "batched": synth.batched,
        "stress": synth.stress}
# typical items and placed boxes of one instance of each family (for work())
_ITEMS = {"single_pass": 90, "multi_restart": 75, "batched": 97, "stress": 196}
_BOXES = {"single_pass": 70, "multi_restart": 60, "batched": 60, "stress": 58}


def listed():
    return [
        # smallest solve: one instance, one greedy decode, latency of a lone request (the
        # benchmark's single_pass workload)
        _solve("single", gen="single_pass", insts=1, restarts=1, eps=0.0, theta=None),
        # the drop-in seat of the reference's per-step backend: a host decode loop with one
        # feasibility launch per item
        {"name": "plain_decode", "kind": "plain", "gen": "multi_restart", "restarts": 1, "eps": 0.3, "theta": 0.9},
        # one instance, many restarts, best of them (the benchmark's multi_restart workload)
        _solve("multi_restart", gen="multi_restart", insts=1, restarts=1024),
        # an ordinary batch: 61 pallets, 48 restarts each, the best of each wanted
        _solve("batch_small", gen="batched", insts=61, restarts=48, best_only=True),
        # the largest batch: the benchmark's default workload, every restart kept
        _solve("batch_full", gen="batched", insts=4096, restarts=256),
        # many box types, partial rotation flags: most steps change the type
        _solve("stress", gen="stress", insts=64, restarts=512, best_only=True),
        # one pallet, several passes per restart, items in input order, another friction and threshold
        _solve("multi_pass", gen="batched", insts=1, restarts=888, passes=4, order="input", mu=0.45, theta=0.5,
               best_only=True),
        # a burst of served requests with the serving workload's restart budgets (64, 256, 1024)
        {"name": "requests", "kind": "serve", "gen": "batched", "requests": 256, "eps": 0.3, "theta": 0.9},
        # the block-building engine in its campaign configuration (the benchmark's block workload)
        _block("block", insts=512, restarts=64),
        # one check of a mid-decode state: extreme points of 48 placed boxes, one box type
        {"name": "feas_step", "kind": "feas", "state": "decode", "boxes": 48, "cand": 230, "ors": 6},
        # one check of stress size (the benchmark's feas workload): 4096 points, 512 boxes
        {"name": "feas_large", "kind": "feas", "state": "grid", "boxes": 512, "cand": 4096, "ors": 6},
        # decode into the caller's device buffers without allocating, every restart returned
        {"name": "noalloc", "kind": "noalloc", "gen": "batched", "restarts": 500, "eps": 0.3, "theta": 0.9},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve"] * 5 + ["block", "feas", "plain", "noalloc", "serve"])
    if kind == "solve":
        gen = rng.choice(["single_pass", "multi_restart", "batched", "batched", "stress"])
        most = 300000 if gen == "stress" else 600000   # decodes of one call
        insts = log(1, 3000)
        restarts = log(1, min(4096, max(1, most // insts)))
        passes = 1
        if rng.random() < 0.25:   # a pallet given more passes is solved on its own
            insts, passes = 1, rng.randint(2, 5)
        c = _solve(None, gen=gen, insts=insts, restarts=restarts, passes=passes,
                   eps=rng.choice([0.0, 0.1, 0.3, 0.3, 0.6]), theta=rng.choice([0.9, 0.9, 0.5, None]),
                   order=rng.choice(["volume", "volume", "volume", "input"]),
                   mu=rng.choice([0.2, 0.2, 0.45]), best_only=rng.random() < 0.5)
    elif kind == "block":
        insts = log(1, 600)
        c = _block(None, insts=insts, restarts=log(1, max(2, min(512, 60000 // insts))),
                   pick=rng.choice(["first", "first", "support", "contact"]))
    elif kind == "feas":
        if rng.random() < 0.5:
            boxes = rng.randint(1, 70)
            c = {"kind": "feas", "state": "decode", "boxes": boxes, "cand": rng.randint(1, 5 * boxes + 3),
                 "ors": rng.choice([1, 2, 4, 6])}
        else:
            c = {"kind": "feas", "state": "grid", "boxes": log(16, 2000), "cand": log(64, 20000),
                 "ors": rng.choice([1, 2, 4, 6])}
    elif kind == "serve":
        c = {"kind": "serve", "gen": "batched", "requests": log(4, 600), "eps": 0.3, "theta": 0.9}
    else:
        c = {"kind": kind, "gen": rng.choice(["single_pass", "multi_restart", "batched"]),
             "restarts": log(1, 3) if kind == "plain" else log(1, 4000), "eps": rng.choice([0.0, 0.3]),
             "theta": rng.choice([0.9, None])}
    return c


def _solve(name, gen, insts, restarts, passes=1, eps=0.3, theta=0.9, order="volume", mu=0.2, best_only=False):
    c = {"name": name, "kind": "solve", "gen": gen, "insts": insts, "restarts": restarts, "passes": passes, "eps": eps,
         "theta": theta, "order": order, "mu": mu, "best_only": best_only}
    return c if name else {k: v for k, v in c.items() if k != "name"}


def _block(name, insts, restarts, pick="first"):
    c = {"name": name, "kind": "block", "gen": "batched", "insts": insts, "restarts": restarts, "pick": pick}
    return c if name else {k: v for k, v in c.items() if k != "name"}


def _base(seed):
    return 100000 + (int(seed) % 1000003) * 4099


def _synth(case, seed, n):
    b = _base(seed)
    return [_GEN[case["gen"]](b + i) for i in range(n)]


def _rows(s):
    return [(t.l, t.lf, t.w, t.wf, t.h, t.hf, t.qty) for t in s.types]


def _instances(case, seed, n):
    return [P.Instance.from_types(s.L, s.W, s.H, _rows(s)) for s in _synth(case, seed, n)]


def _opts(case, seed):
    """Run options; restart seeds start at 0 as in the benchmark workloads."""
    if case["kind"] == "block":
        return P.make_opts(seed=0, restarts=case["restarts"], eps=0.5, theta=0.9, engine="block", amax=4, bmax=4,
                           kmax=6, topk=64, pick=case["pick"])
    return P.make_opts(seed=0, restarts=case["restarts"], passes=case.get("passes", 1), eps=case["eps"],
                       theta=case["theta"], order=case.get("order", "volume"), mu=case.get("mu", 0.2),
                       best_only=case.get("best_only", False))


_server = []


def _serving_handle():
    """The one handle a serving program keeps: its persistent launch holds the
    SMs while requests are in flight, so states do not each get one."""
    if not _server:
        _server.append(P.Handle())
    return _server[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "block"):
        insts = _instances(case, seed, case["insts"])
        return {"kind": kind, "handle": P.Handle(), "insts": insts, "opts": _opts(case, seed)}
    if kind == "serve":
        rng = random.Random(seed)
        insts = _instances(case, seed, case["requests"])
        opts = [P.make_opts(seed=0, restarts=rng.choice((64, 256, 1024)), eps=case["eps"], theta=case["theta"])
                for _ in insts]
        return {"kind": kind, "handle": _serving_handle(), "insts": insts, "opts": opts}
    if kind == "plain":
        return {"kind": kind, "insts": _instances(case, seed, 1), "restarts": case["restarts"], "eps": case["eps"],
                "theta": case["theta"]}
    if kind == "noalloc":
        # buffers of a program that takes instances of up to 512 items
        inst = next(i for i in _instances(case, seed, 64) if i.info()[2] <= 512)
        return {"kind": kind, "insts": [inst], "opts": _opts(case, seed),
                "heads": torch.zeros(case["restarts"], 4, dtype=torch.int64, device="cuda"),
                "places": torch.zeros(case["restarts"] * 512, dtype=torch.int64, device="cuda")}
    cand, ors, boxes = _step(case, seed)
    return {"kind": kind, "cand": torch.tensor(cand, dtype=torch.int32).cuda(),
            "ors": torch.tensor(ors, dtype=torch.int32).cuda(), "boxes": torch.tensor(boxes, dtype=torch.int32).cuda(),
            "bits": torch.zeros(len(cand) * len(ors), dtype=torch.uint8, device="cuda")}


def run(state):
    kind = state["kind"]
    if kind in ("solve", "block"):
        return _best(state["handle"].solve(state["insts"], state["opts"]))
    if kind == "serve":
        h = state["handle"]
        ids = [h.submit(i, o) for i, o in zip(state["insts"], state["opts"])]
        results = []
        for rid in ids:
            if h.wait(rid) != P.OK:
                raise RuntimeError(P.last_error(h._p))
            results.append(h.take(rid))
        return _best(results)
    if kind == "plain":
        r = P.run_plain(state["insts"][0], seed=0, restarts=state["restarts"], eps=state["eps"], theta=state["theta"])
        return _best([r])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "noalloc":
        _ok(P.lib().plp_decode_noalloc(state["insts"][0]._p, ctypes.byref(state["opts"]),
                                       ctypes.c_void_p(state["heads"].data_ptr()),
                                       ctypes.c_void_p(state["places"].data_ptr()), stream))
        return {"heads": state["heads"], "places": state["places"]}
    cand, ors, boxes, bits = state["cand"], state["ors"], state["boxes"], state["bits"]
    _ok(P.lib().plp_feas_check_all_dev(ctypes.c_void_p(cand.data_ptr()), len(cand), ctypes.c_void_p(ors.data_ptr()),
                                       len(ors), ctypes.c_void_p(boxes.data_ptr()), len(boxes), L, W, H,
                                       ctypes.c_void_p(bits.data_ptr()), stream))
    return bits


def _ok(status):
    if status != P.OK:
        raise RuntimeError(P.last_error())


def _row_room(n):
    """Placement rows kept for n packings (about 60 each, the densest about 400)."""
    return 160 * n + 4000


def _best(results):
    """The best packing of every result: (restart, fallback, boxes, passes,
    volume, score) and its placement rows, those of all results one after the
    other, zero rows behind them. Read with the C calls straight into arrays,
    as a compiled program would."""
    lib, n = P.lib(), len(results)
    best, fb, boxes, passes = (np.zeros(n, np.int32) for _ in range(4))
    volume, score = np.zeros(n, np.int64), np.zeros(n, np.float64)
    rows = np.zeros((_row_room(n), 7), np.int32)
    at, used, s = rows.ctypes.data, 0, P.Summary()
    k, f, m = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
    pk, pf, pm, ps = ctypes.byref(k), ctypes.byref(f), ctypes.byref(m), ctypes.byref(s)
    for i, r in enumerate(results):
        _ok(lib.plp_result_best(r._p, pk, pf))
        _ok(lib.plp_result_summary(r._p, k.value, ps))
        _ok(lib.plp_result_placements(r._p, k.value, at + 28 * used, len(rows) - used, pm))
        used += m.value
        best[i], fb[i], boxes[i], passes[i] = k.value, f.value, s.n_boxes, s.n_passes
        volume[i], score[i] = s.volume, s.score
    return {"best": best, "fallback": fb, "n_boxes": boxes, "n_passes": passes, "volume": volume, "score": score,
            "rows": rows}


def work(case):
    """Bytes: instance tables in, what the call returns out. Operations: every
    item step looks at every live point once (about 2.4 per placed box over
    a decode, six compares each); a feasibility check looks at every
    (point, box) pair once."""
    if case["kind"] == "feas":
        n = case["cand"]
        return {"bytes": 12 * n + 24 * case["boxes"] + n * case["ors"], "flops": 6.0 * n * case["boxes"]}
    gen = case["gen"]
    insts = case.get("insts", case.get("requests", 1))
    restarts = case.get("restarts", 448)
    decodes = float(insts) * restarts * case.get("passes", 1)
    kept = insts if case.get("best_only") else insts * restarts
    tables = insts * (88 * 30 + 4 * _ITEMS[gen])
    return {"bytes": float(tables + 32 * insts * restarts + 8 * _BOXES[gen] * kept),
            "flops": decodes * _ITEMS[gen] * 6 * 2.4 * _BOXES[gen]}


# ---------------------------------------------------------------------------
# inputs of the one-step check, and the plain Python decoder behind exact()
# ---------------------------------------------------------------------------
def _step(case, seed):
    """(points, orientations, placed boxes) of one feasibility check."""
    rng = random.Random(_base(seed))
    n, n_cand = case["boxes"], case["cand"]
    if case["state"] == "decode":
        # a decode's state: a first-fit packing of a batched instance and its extreme points
        boxes, b = [], _base(seed)
        while len(boxes) < n:
            boxes, b = _Plain(synth.batched(b)).decode(None, 0.0, stop=n)[1], b + 1
        dims = (rng.randint(15, 50), rng.randint(15, 50), rng.randint(15, 50))
        pts = [(0, 0, 0)]
        for x, y, z, x2, y2, z2 in boxes:
            pts = _extend(pts, x, y, z, x2, y2, z2)
        pts = set(rng.sample(pts, min(len(pts), n_cand)))
        top = H
    else:
        # boxes in layers on a grid of columns; their corners, and points anywhere among them
        cols = [(x, y) for x in range(0, L - 40, 41) for y in range(0, W - 40, 41)]
        rng.shuffle(cols)
        boxes = []
        for i in range(n):
            x, y = cols[i % len(cols)]
            z = 11 * (i // len(cols))
            boxes.append((x, y, z, x + rng.randint(10, 40), y + rng.randint(10, 40), z + rng.randint(5, 11)))
        pts = sorted({(x, y, z) for b in boxes for x in (b[0], b[3]) for y in (b[1], b[4]) for z in (b[2], b[5])})
        pts, top = set(rng.sample(pts, min(len(pts), n_cand))), min(H, 11 * (n // len(cols) + 2))
        dims = (rng.randint(10, 60), rng.randint(10, 60), rng.randint(10, 60))
    while len(pts) < n_cand:
        pts.add((rng.randrange(L), rng.randrange(W), rng.randrange(top)))
    cand = sorted(pts, key=lambda p: (p[2], p[1], p[0]))
    a, b, c = dims
    ors = [(b, c, a), (c, b, a), (a, c, b), (c, a, b), (a, b, c), (b, a, c)][:case["ors"]]
    return cand, ors, boxes


def _extend(cand, x, y, z, x2, y2, z2):
    """Extreme points after a box: those strictly inside go, its corners come."""
    pts = {p for p in cand if not (x < p[0] < x2 and y < p[1] < y2 and z < p[2] < z2)}
    pts.update((px, py, pz) for px in (x, x2) for py in (y, y2) for pz in (z, z2))
    return sorted(pts, key=lambda p: (p[2], p[1], p[0]))


class _Plain:
    """The extreme-point decoder in plain Python, one instance."""

    def __init__(self, s):
        self.ors, seq = [], []
        for i, t in enumerate(s.types):
            o = []
            for flag, pair in ((t.lf, ((t.w, t.h, t.l), (t.h, t.w, t.l))), (t.wf, ((t.l, t.h, t.w), (t.h, t.l, t.w))),
                               (t.hf, ((t.l, t.w, t.h), (t.w, t.l, t.h)))):
                if flag:
                    o += [d for d in pair if d not in o]
            self.ors.append(list(dict.fromkeys(o)))
            seq += [(-t.volume, i, c) for c in range(t.qty)]
        self.input_order = [i for _, i, _ in seq]
        self.volume_order = [i for _, i, _ in sorted(seq)]

    def decode(self, rng, eps, order="volume", stop=None):
        """One pass: (placement rows, placed boxes)."""
        cand, rows, boxes = [(0, 0, 0)], [], []
        for t in self.input_order if order == "input" else self.volume_order:
            if stop is not None and len(boxes) >= stop:
                break
            feas = []
            for x, y, z in cand:
                for d in self.ors[t]:
                    if self._fits(x, y, z, d, boxes):
                        feas.append((x, y, z) + d)
                        if eps == 0.0:
                            break
                if feas and eps == 0.0:
                    break
            if not feas:
                continue
            p = feas[0]
            if eps > 0.0 and rng.random() >= 1.0 - eps:
                p = feas[rng.randrange(len(feas))]
            x, y, z, w, d, h = p
            rows.append((t,) + p)
            boxes.append((x, y, z, x + w, y + d, z + h))
            cand = _extend(cand, *boxes[-1])
        return rows, boxes

    @staticmethod
    def _fits(x, y, z, wdh, boxes):
        x2, y2, z2 = x + wdh[0], y + wdh[1], z + wdh[2]
        if x2 > L or y2 > W or z2 > H:
            return False
        area = 0
        for b in boxes:
            if b[0] < x2 and x < b[3] and b[1] < y2 and y < b[4]:
                if b[2] < z2 and z < b[5]:
                    return False
                if b[5] == z:
                    area += (min(x2, b[3]) - max(x, b[0])) * (min(y2, b[4]) - max(y, b[1]))
        return z == 0 or not area / (wdh[0] * wdh[1]) < 0.5

    @staticmethod
    def score(boxes, mu):
        """Share of boxes whose friction stability ratio is at least 1."""
        n = len(boxes)
        if not n:
            return 0.0
        mass = [50.0 * ((b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2])) / 1e6 for b in boxes]
        load = list(mass)
        for k in sorted(range(n), key=lambda i: (-boxes[i][2], i)):
            b = boxes[k]
            if b[2] == 0:
                continue
            on = []
            for j, c in enumerate(boxes):
                ox, oy = min(b[3], c[3]) - max(b[0], c[0]), min(b[4], c[4]) - max(b[1], c[1])
                if c[5] == b[2] and ox > 0 and oy > 0:
                    on.append((j, ox * oy))
            total = sum(a for _, a in on)
            for j, a in on:
                load[j] += load[k] * a / total
        return sum((mu / 0.3) * f / m >= 1.0 for f, m in zip(load, mass)) / n

    def restart(self, seed, case):
        """(accepted, volume, boxes, score, rows) of one restart's best pass."""
        rng, best = random.Random(seed), None
        theta = case["theta"]
        for _ in range(case.get("passes", 1)):
            rows, boxes = self.decode(rng, case["eps"], case.get("order", "volume"))
            score = self.score(boxes, case.get("mu", 0.2))
            got = (theta is None or score >= theta, sum(r[4] * r[5] * r[6] for r in rows), len(rows), score, rows)
            if best is None or got[:3] > best[:3]:
                best = got
        return best


def exact(case, seed):
    """The answer of the plain Python decoder, where a few decodes are all the
    case does (about a third of a second each)."""
    if case["kind"] not in ("solve", "plain"):
        return None
    insts = case.get("insts", 1)
    if insts * case["restarts"] * case.get("passes", 1) * (3 if case["gen"] == "stress" else 1) > 16:
        return None
    out = []
    for s in _synth(case, seed, insts):
        plain, best = _Plain(s), None
        for k in range(case["restarts"]):
            got = plain.restart(k, case)
            if best is None or got[:3] > best[1][:3]:
                best = (k, got)
        out.append(best)
    passes = case.get("passes", 1)
    rows = np.zeros((_row_room(len(out)), 7), np.int32)
    placed = [r for _, g in out for r in g[4]]
    rows[:len(placed)] = np.array(placed, np.int32).reshape(-1, 7)
    return {"best": np.array([k for k, _ in out], np.int32), "fallback": np.array([not g[0] for _, g in out], np.int32),
            "n_boxes": np.array([g[2] for _, g in out], np.int32), "n_passes": np.full(len(out), passes, np.int32),
            "volume": np.array([g[1] for _, g in out], np.int64), "score": np.array([g[3] for _, g in out], np.float64),
            "rows": rows}
