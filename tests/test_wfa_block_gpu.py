"""Pairs of large distance on whole blocks: distances on both sides of the warp
kernels' caps (255 plain, 511 routed) and of smax, byte-compared pairs, empty
sides, and walks past several loads of wavefront rows, against the oracle."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, cost_model, workloads
from helpers import assert_wfa_equal, wfa_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pairs():
    rng = np.random.default_rng(57)
    ps, ts = [], []
    for k in range(28):
        s = workloads.random_bases(rng, int(rng.integers(900, 1500)))
        ps.append(s.tobytes())
        ts.append(workloads.mutate_runs(rng, s, 0.02 + 0.02 * k, (1 / 3, 1 / 3, 1 / 3), geom_p=0.5).tobytes())
    for k in (3, 9, 15, 21, 27):                          # byte compare
        ts[k] = ts[k][:100] + b"N" + ts[k][101:]
    s = workloads.random_bases(rng, 700)
    for t in (s[:180], s[-190:], np.concatenate([s, workloads.random_bases(rng, 512)]), s[:0], s):
        ps += [s.tobytes(), t.tobytes()]
        ts += [t.tobytes(), s.tobytes()]
    return ps, ts


@pytest.mark.parametrize("smax", [255, 256, 511, 512, 1100])
@pytest.mark.parametrize("learned", [False, True])
def test_block_pairs_match_oracle(pairs, smax, learned):
    assert cost_model.load_default()
    ps, ts = pairs
    want = oracle.wfa_batch(ps, ts, smax=smax, with_cigar=True, max_smax=4096)
    if smax > 600:
        assert ((want.score > 255) & (want.score < 512)).sum() >= 3 and (want.score > 511).sum() >= 3
    got = wfa_gpu(ps, ts, smax=smax, max_smax=4096, learned=learned)
    assert_wfa_equal(got, want, f"smax {smax}, learned {learned}")
    score = wfa_gpu(ps, ts, smax=smax, with_cigar=False, max_smax=4096, learned=learned)
    assert np.array_equal(score.res["score"], want.score)


@pytest.mark.parametrize("copies", [1, 64])
def test_block_kernel_beside_the_warps_and_after_them(pairs, copies):
    """The largest smax: the stacks of few pairs fit for both kernels at once, those of
    2,432 pairs do not, so there the kernels run one after the other."""
    assert cost_model.load_default()
    ps, ts = pairs
    want = oracle.wfa_batch(ps, ts, smax=3500, with_cigar=True, max_smax=4096)
    got = wfa_gpu(ps * copies, ts * copies, smax=3500, max_smax=4096, learned=True)
    assert np.array_equal(got.res["score"], np.tile(want.score, copies))
    for k in range(len(ps)):
        for c in (0, copies - 1):
            assert got.cigar(c * len(ps) + k) == want.cigars[k], (copies, c, k)
