"""The route pass with 1 to 16 lanes a side: its queue items, lower bounds and the
call's results are those of the batch tiled to one lane a side."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, cost_model, workloads
from helpers import packed

pytestmark = pytest.mark.gpu


def _pairs():
    rng = np.random.default_rng(77)
    ps, ts = [], []
    for n in (0, 1, 2, 3, 100, 255, 256, 257, 258, 259, 260, 511, 515, 1000, 2049, 4100, 4500):
        s = workloads.random_bases(rng, n)
        for rate in (0.02, 0.15):
            t = workloads.mutate_runs(rng, s, rate, (1 / 3, 1 / 3, 1 / 3)) if n else workloads.random_bases(rng, 7)
            ps.append(s.tobytes())
            ts.append(t.tobytes())
    return ps, ts


def _items(torch, ps, ts):
    q = packed(ps, ts)
    batch = api.DeviceBatchT(q.a_buf, q.a_off, q.a_len, q.b_buf, q.b_off, q.b_len)
    n = len(ps)
    score, length = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    cigar = torch.zeros(batch.out_bytes, dtype=torch.uint8, device="cuda")
    api.wfa_device(batch, 64, True, score, length, cigar, learned=True)
    return api.wfa_route_items(n), score.cpu().numpy()


@pytest.mark.parametrize("copies", [1, 40, 160, 300, 600])
def test_route_items_do_not_depend_on_the_lanes(copies):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    ps, ts = _pairs()
    want, score = _items(torch, ps * 1200, ts * 1200)          # 40,800 pairs: one lane a side
    got, s = _items(torch, ps * copies, ts * copies)
    assert np.array_equal(np.asarray(got), np.asarray(want)[: len(got)])
    assert np.array_equal(s, score[: len(s)])
    ref = oracle.wfa_batch(ps, ts, smax=64, with_cigar=False)
    assert np.array_equal(score[: len(ps)], ref.score)
