"""Plain WFA batches of many pairs around the edits at which a pair moves on (255 on a
warp, 511 or smax in the second pass, blocks), with few and with many pairs left by
the first pass, against the oracle."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, workloads

pytestmark = pytest.mark.gpu


def _pairs(long_every, n=3600):
    """n pairs, more than eight a resident block of the device; one in long_every is long."""
    rng = np.random.default_rng(91)
    pats, txts = [], []
    for k in range(n):
        if k % long_every:
            length, rate = int(rng.integers(40, 120)), rng.uniform(0.0, 0.3)
        elif k % 30:
            length, rate = int(rng.integers(500, 800)), rng.uniform(0.45, 0.7)
        else:
            length, rate = int(rng.integers(1200, 1900)), rng.uniform(0.2, 0.7)
        p = workloads.random_bases(rng, length)
        t, _ = workloads.mutate_point(rng, p, np.array([length]), float(rate), (0.6, 0.2, 0.2))
        pats.append(p.tobytes())
        txts.append(t.tobytes())
    for k in (0, 30, 31):
        txts[k] = txts[k][:-3] + b"NNN"                 # bytes instead of 2-bit codes
    return pats, txts


@pytest.mark.parametrize("long_every", [1, 30], ids=["many left", "few left"])
@pytest.mark.parametrize("smax", [512, 700, 701, 900])
@pytest.mark.parametrize("trace", [True, False])
def test_plain_batches_of_many_pairs(smax, trace, long_every):
    torch = pytest.importorskip("torch")
    pats, txts = _pairs(long_every)
    want = oracle.wfa_batch(pats, txts, smax=smax, with_cigar=True, max_smax=4096)
    left = (want.score < 0) | (want.score > 255)
    assert (left.sum() > 2500) == (long_every == 1) and left.sum() > 40
    assert (want.score < 0).any() and ((want.score > 511).any() or smax == 512)
    ps = workloads.from_lists("cap", pats, txts)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cuda")
    sc, ln = (torch.full((b.n,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    cg = torch.zeros(b.out_bytes, dtype=torch.uint8, device="cuda")
    api.wfa_device(b, smax, trace, sc, ln, cg)
    assert np.array_equal(sc.cpu().numpy(), want.score)
    if trace:
        ends = b.out_off.cpu().numpy() + b.a_len.cpu().numpy().astype(np.int64) + b.b_len.cpu().numpy()
        ln, cg = ln.cpu().numpy(), cg.cpu().numpy()
        for i, c in enumerate(want.cigars):
            assert ln[i] == len(c) and cg[ends[i] - len(c):ends[i]].tobytes() == c, i
