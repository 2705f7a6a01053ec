"""Prepared batches whose tables are gone: a run that failed gave them back."""
import pytest

import oracle_py as O
import plpb200 as P
from plpb200 import synth

pytestmark = pytest.mark.gpu


def test_a_batch_whose_run_failed_refuses_to_run_again():
    text = synth.multi_restart(2).to_thpack()
    inst, opts = P.Instance.parse(text), P.make_opts(seed=0, restarts=8)
    with P.Handle() as h:
        h.set_tile(P=128, C=384, G=2, D=1, M=1)
        b = h.prepare([inst], opts)
        b.run()
        b.fetch()
        h.debug_sync_bound(wait_limit=256, skip_warp=1)   # a barrier wait runs out
        with pytest.raises(P.PlpError) as e:
            b.run()
        assert e.value.status == P.E_DEVICE
        h.debug_sync_bound(0, -1)
        for again in (b.run, b.fetch):
            with pytest.raises(P.PlpError) as e:
                again()
            assert e.value.status == P.E_INVALID
        b.close()
        b = h.prepare([inst], opts)
        b.run()
        r = b.fetch()[0]
        for k in range(8):
            assert O.strip_time(r.json(k)) == O.strip_time(O.run(O.OInstance(text), seed=k)[0])
        b.close()


def test_a_batch_may_outlive_its_handle():
    text = synth.multi_restart(2).to_thpack()
    inst, opts = P.Instance.parse(text), P.make_opts(seed=0, restarts=8)
    left = []
    for _ in range(3):
        with P.Handle() as h:
            b = h.prepare([inst], opts)
            b.run()
            r = b.fetch()[0]
            left.append(b)
    for b in left:
        for call in (b.run, b.fetch):
            with pytest.raises(P.PlpError) as e:
                call()
            assert e.value.status == P.E_INVALID
        assert not b.graph
    left.clear()                                          # freed after their handles
    with P.Handle() as h:
        again = h.solve([inst], opts)[0]
    for k in range(8):
        assert O.strip_time(r.json(k)) == O.strip_time(again.json(k)) == O.strip_time(O.run(O.OInstance(text), seed=k)[0])
