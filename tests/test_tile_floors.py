"""Tiles deepened by a batch that outgrew its own (csrc/tile_floor.hpp): the
deeper tile holds for batches of its kind and size, and falls again."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "plp-gpu_b200", "csrc")


def test_floors_are_of_a_kind_bounded_and_fall(tmp_path):
    exe = str(tmp_path / "tile_floor_model")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, "-o", exe, os.path.join(HERE, "tile_floor_model.cpp")],
                   check=True)
    lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    assert lines == ["0 0", "1024 1536", "0 0", "0 0",      # [engine][one wave, several]
                     "32 160", "1024 1536",                 # 20 steps: 32 boxes, 7 x 20 + 1 points
                     "1024 1536", "1024 1536", "0 0"]


@pytest.mark.gpu
def test_an_odd_instance_is_forgotten_and_a_prepared_batch_remembers():
    """600 cubes outgrow the deepest tile chosen from sizes (512 boxes in one
    wave): the run takes a retry, the like of it none for a while."""
    import oracle_py as O
    import plpb200 as P
    from plpb200 import synth

    odd_text = "1\n1 1\n587 233 220\n1\n1 10 1 10 1 10 1 600\n"
    odd = P.Instance.parse(odd_text)
    plain = P.Instance.parse(synth.single_pass(1).to_thpack())
    opts = P.make_opts(seed=5, restarts=2)
    with P.Handle() as h:
        kept = h.prepare([odd], opts)
        first = kept.run()[2]
        assert first > 2                                  # decoder and selection, and the retries'
        again = h.prepare([odd], opts)
        assert again.run()[2] == 2
        for _ in range(70):
            h.solve([plain], opts)
        later = h.prepare([odd], opts)
        assert later.run()[2] == first                    # the handle has forgotten
        assert kept.run()[2] == 2                         # the batch has not
        r = kept.fetch()[0]
        for k in range(2):
            assert O.strip_time(r.json(k)) == O.strip_time(O.run(O.OInstance(odd_text), seed=5 + k)[0])
        for b in (kept, again, later):
            b.close()
