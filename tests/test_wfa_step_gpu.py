"""The WFA forward pass and walk at their edges: lengths around the 16-base words
the extension compares, smax equal to the distance and one below it (the
wavefronts narrow towards the final diagonal as edits run out), a final diagonal
at +-smax, one side much shorter than smax (the wavefront is clipped to the
matrix), and walks longer than the rows loaded at once, for every group size."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, cost_model, workloads
from helpers import assert_wfa_equal, wfa_gpu

pytestmark = pytest.mark.gpu


def _pairs(seed):
    rng = np.random.default_rng(seed)
    ps, ts = [], []
    for n in (1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 160, 257):
        s = workloads.random_bases(rng, n)
        for t in (s, workloads.mutate_runs(rng, s, 0.1, (1 / 3, 1 / 3, 1 / 3), 0.5),
                  workloads.mutate_runs(rng, s, 0.3, (1 / 3, 1 / 3, 1 / 3)), s[: n // 2], s[n // 3:],
                  np.concatenate([s, workloads.random_bases(rng, 24)]),
                  np.concatenate([workloads.random_bases(rng, 25), s]), workloads.random_bases(rng, n)):
            ps.append(s.tobytes())
            ts.append(t.tobytes())
            ps.append(t.tobytes())
            ts.append(s.tobytes())
    for k in range(0, len(ts), 11):                       # byte compare instead of 2-bit codes
        ts[k] = ts[k][: len(ts[k]) // 2] + b"N" + ts[k][len(ts[k]) // 2 + 1:]
    return ps, ts


@pytest.mark.parametrize("smax", [0, 1, 5, 24, 25, 64, 100])
def test_plain_matches_oracle(smax):
    ps, ts = _pairs(31)
    want = oracle.wfa_batch(ps, ts, smax=smax, with_cigar=True)
    assert_wfa_equal(wfa_gpu(ps, ts, smax=smax), want, f"smax {smax}")
    score = wfa_gpu(ps, ts, smax=smax, with_cigar=False)
    assert np.array_equal(score.res["score"], want.score)


@pytest.mark.parametrize("group", [8, 16, 32])
def test_groups_match_oracle(group):
    assert cost_model.load_default()
    ps, ts = _pairs(32)
    before = api.tune_get()
    try:
        api.tune_set(wfa_lane_smax=0, wfa_group=group)
        for smax in (5, 24, 100):
            want = oracle.wfa_batch(ps, ts, smax=smax, with_cigar=True)
            assert_wfa_equal(wfa_gpu(ps, ts, smax=smax, learned=True), want, f"group {group}, smax {smax}")
    finally:
        api.tune_set(**before)


def test_smax_at_the_distance():
    """Each pair alone, resolved at smax = its distance and not one below."""
    ps, ts = _pairs(33)
    d = oracle.wfa_batch(ps, ts, smax=300, with_cigar=False).score
    for k in range(0, len(ps), 7):
        if not ps[k] or not ts[k] or d[k] < 1:
            continue
        for smax in (int(d[k]), int(d[k]) - 1):
            want = oracle.wfa_batch(ps[k:k + 1], ts[k:k + 1], smax=smax, with_cigar=True)
            assert_wfa_equal(wfa_gpu(ps[k:k + 1], ts[k:k + 1], smax=smax), want, f"pair {k}, smax {smax}")


@pytest.mark.parametrize("copies", [1, 60])
def test_one_and_two_diagonals_a_lane(copies):
    """The warp queue with no more pairs than warps (two diagonals a lane) and with more."""
    assert cost_model.load_default()
    ps, ts = _pairs(34)
    ps, ts = ps * copies, ts * copies
    before = api.tune_get()
    try:
        api.tune_set(wfa_lane_smax=0, wfa_group=32)
        want = oracle.wfa_batch(ps, ts, smax=100, with_cigar=True)
        assert_wfa_equal(wfa_gpu(ps, ts, smax=100, learned=True), want, f"{len(ps)} pairs")
    finally:
        api.tune_set(**before)
