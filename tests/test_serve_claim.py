"""Serving decoders' claims (csrc/serve_claim.hpp) on a model of the claim words
whose scheduler holds failed claims back: every published item is claimed, also
by decoders that were told to stop."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "plp-gpu_b200", "csrc")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("claim") / "serve_claim_model")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, "-o", exe,
                    os.path.join(HERE, "serve_claim_model.cpp")], check=True)
    return exe


@pytest.mark.parametrize("mode", ["progress", "stop"])
def test_pending_failures_keep_nobody_from_an_item(model, mode):
    out = subprocess.run([model, mode], capture_output=True, text=True, check=True, timeout=120).stdout
    taken, published, granted = map(int, out.split())
    assert published == 20
    assert taken == published, f"{taken} items after {granted} accesses"


@pytest.mark.parametrize("mode,took,polls", [
    ("main-waits", 1, (20000, 20001)), ("deep-waits", 1, (20000, 20001)),   # the launch was in use all the while
    ("main-idle", 0, (6000, 8000)), ("deep-left", 0, (0, 1))])
def test_decoders_stay_while_the_launch_is_in_use(model, mode, took, polls):
    """An idle bound of 2000 polls, counted from the last claim of the launch."""
    out = subprocess.run([model, mode], capture_output=True, text=True, check=True, timeout=120).stdout
    got, n = map(int, out.split())
    assert got == took
    assert polls[0] <= n <= polls[1]


@pytest.mark.gpu
def test_small_requests_into_an_idle_launch():
    """Requests of 1 to 16 restarts, back to back and one at a time, into a
    launch whose decoders are nearly all idle: none waits for the decoders' idle
    bound (about a second)."""
    import time

    import oracle_py as O
    import plpb200 as P
    from plpb200 import synth

    texts = [synth.single_pass(s).to_thpack() for s in (1, 2)]
    insts = [P.Instance.parse(t) for t in texts]
    with P.Handle() as h:
        def one(q):
            return h.submit(insts[q % 2], P.make_opts(seed=q, restarts=1 + q % 16))

        def done(q, rid):
            assert h.wait(rid, 5000) == P.OK
            return h.take(rid)

        done(0, one(0))                        # set-up of the serving path
        t0 = time.perf_counter()
        res = [done(q, rid) for q, rid in enumerate([one(q) for q in range(400)])]
        assert time.perf_counter() - t0 < 0.7
        worst = 0.0
        for q in range(60):
            t0 = time.perf_counter()
            done(q, one(q))
            worst = max(worst, time.perf_counter() - t0)
        assert worst < 0.7
        assert h.serve_counters()["served"] == 461
    for q in range(0, 400, 57):
        oi = O.OInstance(texts[q % 2])
        for k in range(1 + q % 16):
            assert O.strip_time(res[q].json(k)) == O.strip_time(O.run(oi, seed=q + k)[0])


@pytest.mark.gpu
def test_requests_after_a_long_overflow(monkeypatch):
    """A request whose restarts all outgrow the main decoders' tile keeps two
    overflow decoders busy for longer than the idle bound of about a second.
    Small requests beside it and the next one are served meanwhile and at once
    after it (the overflow decoders' own bound is a minute)."""
    import time

    import oracle_py as O
    import plpb200 as P
    from plpb200 import synth

    monkeypatch.setenv("PLP_SERVE_TILE", "16,32,16")
    monkeypatch.setenv("PLP_SERVE_DEEP", "2")
    big = synth.batched(30003).to_thpack()
    small = "1\n1 1\n100 100 100\n1\n1 50 1 50 1 50 1 8\n"
    bi, si = P.Instance.parse(big), P.Instance.parse(small)
    with P.Handle() as h:
        def served(inst, seed, restarts):
            t = time.perf_counter()
            rid = h.submit(inst, P.make_opts(seed=seed, restarts=restarts))
            assert h.wait(rid, 40000) == P.OK, P.last_error()
            return h.take(rid), time.perf_counter() - t

        served(bi, 0, 1)                       # set-up
        _, one = served(bi, 0, 64)
        n = max(64, min(65536, int(3.0 / max(one, 1e-3) * 64)))   # some three seconds of overflow decodes
        t0 = time.perf_counter()
        rid = h.submit(bi, P.make_opts(seed=1, restarts=n))
        time.sleep(1.6)
        beside = [served(si, q, 4) for q in range(3)]
        during = h.poll(rid) == P.E_PENDING
        assert h.wait(rid, 60000) == P.OK
        long_one, took = h.take(rid), time.perf_counter() - t0
        after, dt = served(bi, 7, 64)
        assert dt < 10
        if during:
            assert all(t < 1.0 for _, t in beside)
    oi, os_ = O.OInstance(big), O.OInstance(small)
    for k in (0, n - 1):
        assert O.strip_time(long_one.json(k)) == O.strip_time(O.run(oi, seed=1 + k)[0])
    assert O.strip_time(after.json(63)) == O.strip_time(O.run(oi, seed=70)[0])
    for q, (r, _) in enumerate(beside):
        assert O.strip_time(r.json(3)) == O.strip_time(O.run(os_, seed=q + 3)[0])
