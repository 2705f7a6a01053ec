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
