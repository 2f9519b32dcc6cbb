"""Letters of SW sequences read by 1 to 32 lanes each: pairs whose only byte outside
A, C, G, T is the last, the first or one at a step's edge are scored as the oracle
scores them (N is a letter of the 16-bit kernels, R of the 32-bit ones alone)."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, workloads

pytestmark = pytest.mark.gpu

SCORING = (2, -3, 3, 1)


# more pairs than the device has threads for a warp each, at mean sizes for each group; and few pairs (a warp)
@pytest.mark.parametrize("n,length", [(200_000, 12), (90_000, 30), (60_000, 100), (24_000, 200), (12_000, 420),
                                      (6_000, 700), (300, 600)])
def test_letters_at_the_edges(n, length):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    lens = rng.integers(max(1, length - 10), length + 10, n)
    ends = np.cumsum(lens)
    sides = [workloads.random_bases(rng, int(ends[-1])) for _ in range(2)]
    sides[1][:] = np.where(rng.random(sides[1].size) < 0.9, sides[0], sides[1])
    first = ends - lens
    for k, letter in enumerate(b"NRnR"):
        for side in sides:
            pick = rng.choice(n, n // 20, replace=False)
            at = (first[pick], ends[pick] - 1, first[pick] + np.minimum(lens[pick] - 1, 15),
                  first[pick] + np.minimum(lens[pick] - 1, 16))[k]
            side[at] = letter
    off, lens = first.astype(np.int64), lens.astype(np.int32)
    b = api.DeviceBatchT(sides[0], off, lens, sides[1], off, lens, device="cuda")
    score, pos = (torch.full((m * n,), -7, dtype=torch.int32, device="cuda") for m in (1, 4))
    api.sw_device(b, SCORING, False, score, pos, None, None)
    want = oracle.sw_batch([sides[0][o:e].tobytes() for o, e in zip(off, ends)],
                           [sides[1][o:e].tobytes() for o, e in zip(off, ends)], scoring=SCORING, with_cigar=False)
    assert np.array_equal(score.cpu().numpy(), want.score)
