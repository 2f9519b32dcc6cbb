"""Smith-Waterman pairs with N: they run on the 16-bit kernels, where N is a
letter of its own (it matches N alone, as the reference's byte comparison has
it); any other byte outside A, C, G, T sends a pair to the 32-bit kernels.  Both
agree with the oracle around the bands' and tiles' edges, alone and paired with
pairs of the other kind."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import workloads
from helpers import assert_sw_equal, sw_gpu

pytestmark = pytest.mark.gpu


def _sprinkle(rng, s, rate, letter):
    s = s.copy()
    s[rng.random(s.shape[0]) < rate] = ord(letter)
    return s


def _pairs(n, seed):
    """Around n columns: N in the text, in the pattern, in both at the same and at
    different places, runs of N, N alone, and other letters beside it."""
    rng = np.random.default_rng(seed)
    ts, ps = [], []
    for cols in (n - 1, n, n + 1):
        p = workloads.random_bases(rng, cols)
        t = np.concatenate([workloads.random_bases(rng, 9), workloads.mutate_runs(rng, p, 0.05, (0.6, 0.2, 0.2)),
                            workloads.random_bases(rng, 5)])
        run_p, run_t = p.copy(), t.copy()
        run_p[cols // 3: cols // 3 + 7] = ord("N")
        run_t[9 + cols // 3: 9 + cols // 3 + 7] = ord("N")
        for a, b in ((_sprinkle(rng, t, 0.1, "N"), p), (t, _sprinkle(rng, p, 0.1, "N")), (run_t, run_p),
                     (_sprinkle(rng, t, 0.3, "N"), _sprinkle(rng, p, 0.3, "N")), (_sprinkle(rng, t, 0.1, "n"), p),
                     (_sprinkle(rng, run_t, 0.05, "R"), run_p), (t, p), (t, np.full(cols, ord("N"), np.uint8)),
                     (np.full(cols + 3, ord("N"), np.uint8), np.full(cols, ord("N"), np.uint8))):
            ts.append(a.tobytes())
            ps.append(b.tobytes())
    return ts, ps


@pytest.mark.parametrize("n", [2, 32, 64, 128, 256, 512, 1100])
@pytest.mark.parametrize("with_cigar", [True, False])
def test_n_pairs_match_oracle(n, with_cigar):
    ts, ps = _pairs(n, 900 + n)
    for scoring in ((2, -3, 3, 1), (2, -3, 5, 2)):
        want = oracle.sw_batch(ts, ps, scoring=scoring, with_cigar=with_cigar)
        assert_sw_equal(sw_gpu(ts, ps, scoring=scoring, with_cigar=with_cigar), want, f"{n} columns, {scoring}")
