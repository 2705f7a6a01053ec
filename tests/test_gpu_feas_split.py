"""The one-step feasibility kernel splits 32 candidates per block and the boxes
over the block's warps: candidate and box counts around those edges, more than
six orientations, coordinates near 2^30, and the host entry's two transfer
paths (small inputs read in place, larger ones copied), against the oracle."""
import ctypes
import random

import numpy as np
import pytest
import torch

import oracle_py as O
import plpb200 as P

pytestmark = pytest.mark.gpu


def _case(rng, n_cand, n_ors, n_fast, base):
    L, W, H = base + 300, base + 200, base + 100
    levels = [0, 10, 20, 40]
    boxes = []
    for _ in range(n_fast):
        x, y, z = base + rng.randint(0, 290), base + rng.randint(0, 190), base * (rng.random() < 0.8) + rng.choice(levels)
        boxes.append((x, y, z, x + rng.randint(1, 60), y + rng.randint(1, 60), z + rng.choice([10, 20])))
    cand = []
    for _ in range(n_cand):
        if boxes and rng.random() < 0.6:
            b = rng.choice(boxes)
            cand.append((rng.choice([b[0], b[3]]), rng.choice([b[1], b[4]]), rng.choice([b[2], b[5]])))
        else:
            cand.append((base + rng.randint(0, 300), base + rng.randint(0, 200), rng.choice([0, base + 10])))
    ors = [(rng.randint(1, 50), rng.randint(1, 50), rng.randint(1, 40)) for _ in range(n_ors)]
    return cand, ors, np.asarray(boxes, np.int32).reshape(-1, 6), (L, W, H)


@pytest.mark.parametrize("base", [0, 1 << 30])
@pytest.mark.parametrize("n_cand,n_ors,n_fast", [(1, 1, 0), (1, 6, 1), (31, 2, 15), (32, 6, 16), (33, 7, 17), (65, 13, 40),
                                                 (700, 6, 300), (3000, 6, 900), (40, 6, 4842)])
def test_feasibility_at_the_split_edges(n_cand, n_ors, n_fast, base):
    cand, ors, boxes, (L, W, H) = _case(random.Random(n_cand * 7 + n_fast), n_cand, n_ors, n_fast, base)
    exp = O.check_all(cand, ors, boxes, L, W, H)
    assert np.array_equal(P.feas_check_all(cand, ors, boxes, L, W, H), exp)
    dev = [torch.tensor(np.asarray(a, np.int32).reshape(-1, k)).cuda() for a, k in ((cand, 3), (ors, 3), (boxes, 6))]
    bits = torch.full((n_cand * n_ors + 1,), 7, dtype=torch.uint8, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) if t.numel() else None for t in dev]
    st = P.lib().plp_feas_check_all_dev(ptr[0], n_cand, ptr[1], n_ors, ptr[2], n_fast, L, W, H,
                                        ctypes.c_void_p(bits.data_ptr()),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == P.OK
    got = bits.cpu().numpy()
    assert np.array_equal(got[:-1], exp) and got[-1] == 7
