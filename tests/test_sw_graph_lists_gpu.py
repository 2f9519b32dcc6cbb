"""Replays of a synchronous ga_sw_device call whose pairs moved, behind the same
pointers, to a work list that was empty when the graph was captured: a pair gains
a letter that the 16-bit kernels do not take, grows past the long shape's
threshold, or past the bound under which its score surely fits 16 bits."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, workloads

pytestmark = pytest.mark.gpu

POS = ("start_i", "start_j", "end_i", "end_j")


def _pairs(seed, n, length, rate=0.03):
    rng = np.random.default_rng(seed)
    ts, ps = [], []
    for _ in range(n):
        p = workloads.random_bases(rng, length)
        t, _ = workloads.mutate_point(rng, p, np.array([length]), rate, (0.6, 0.2, 0.2))
        t = np.concatenate([t, workloads.random_bases(rng, length)])[:length]
        ts.append(t.tobytes())
        ps.append(p.tobytes())
    return ts, ps


def _outs(torch, batch):
    outs = [torch.full((k * batch.n,), -7, dtype=torch.int32, device="cuda") for k in (1, 4, 1)]
    return outs + [torch.zeros(max(batch.out_bytes, 1), dtype=torch.uint8, device="cuda")]


def _call(torch, batch, scoring, outs, want, label):
    for t in outs:
        t.fill_(-7 if t.dtype == torch.int32 else 0)
    torch.cuda.synchronize()
    api.sw_device(batch, scoring, True, *outs, stream=None, trace_cell_limit=1 << 30)
    sc, pos, ln, cg = (t.cpu().numpy() for t in outs)
    assert np.array_equal(sc, want.score), label
    for k, f in enumerate(POS):
        assert np.array_equal(pos.reshape(-1, 4)[:, k], getattr(want, f)), (label, f)
    ends = batch.out_off.cpu().numpy() + batch.a_len.cpu().numpy().astype(np.int64) + batch.b_len.cpu().numpy()
    for i, c in enumerate(want.cigars):
        assert int(ln[i]) == len(c) and cg[ends[i] - len(c):ends[i]].tobytes() == c, (label, i)


def _device(ts, ps):
    s = workloads.from_lists("lists", ts, ps)
    return api.DeviceBatchT(s.a_buf, s.a_off, s.a_len, s.b_buf, s.b_off, s.b_len, device="cuda")


def _oracle(ts, ps, scoring):
    return oracle.sw_batch(ts, ps, scoring=scoring, with_cigar=True, trace_cell_limit=1 << 30)


@pytest.mark.parametrize("n", [7, 5000])
def test_pair_gains_a_letter_of_no_16_bit_kernel(n):
    torch = pytest.importorskip("torch")
    scoring = (2, -3, 3, 1)
    ts, ps = _pairs(61, n, 120)
    batch = _device(ts, ps)
    outs, want = _outs(torch, batch), _oracle(ts, ps, scoring)
    for rep in range(3):
        _call(torch, batch, scoring, outs, want, ("ACGT", rep))
    k = n // 2
    ts[k] = ts[k][:50] + b"R" + ts[k][51:]
    batch.seq[int(batch.a_off[k]) + 50] = ord("R")
    want = _oracle(ts, ps, scoring)
    for rep in range(3):
        _call(torch, batch, scoring, outs, want, ("R", rep))


def _grown(torch, scoring, short, full, n):
    """Three calls on the pairs' first `short` bases, then on all `full` of them."""
    ts, ps = _pairs(62, n, full)
    batch = _device(ts, ps)
    a, b = batch.a_len.clone(), batch.b_len.clone()
    batch.a_len.clamp_(max=short)
    batch.b_len.clamp_(max=short)
    cut = [t[:short] for t in ts], [p[:short] for p in ps]
    outs, want = _outs(torch, batch), _oracle(*cut, scoring)
    for rep in range(3):
        _call(torch, batch, scoring, outs, want, ("short", rep))
    batch.a_len.copy_(a)
    batch.b_len.copy_(b)
    want = _oracle(ts, ps, scoring)
    for rep in range(3):
        _call(torch, batch, scoring, outs, want, ("grown", rep))


def test_pairs_grow_past_the_long_shape_threshold():
    # (a scheme of no 16-bit kernel: every pair is in a 32-bit list)
    _grown(pytest.importorskip("torch"), (2, -9, 3, 1), 300, 4200, 6)


def test_pairs_grow_past_the_16_bit_score_bound():
    """Pairs of 2,000 bases score some 37,000 at 20 a match: taken on the
    optimistic rule, they overflow 16 bits and are handed over."""
    torch = pytest.importorskip("torch")
    before = api.tune_get()
    try:
        api.tune_set(sw_opt16_pct=70)
        _grown(torch, (20, -30, 30, 10), 1200, 2000, 6)
    finally:
        api.tune_set(**before)
