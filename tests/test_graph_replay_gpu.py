"""Calls that repeat run as CUDA graph replays: the same shape three times in a
row, through each entry, with other sequences of equal lengths behind the same
buffers before the third, equals the oracle every time; a call that differs in
one buffer alone is not served by the graph of the other."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, cost_model, workloads

pytestmark = pytest.mark.gpu

SCORING = (2, -3, 3, 1)
POS = ("start_i", "start_j", "end_i", "end_j")


def _substituted(seed, lens, rates):
    """(patterns, texts) of the given lengths: texts are the patterns with substitutions at each pair's rate."""
    rng = np.random.default_rng(seed)
    pats, txts = [], []
    for length, rate in zip(lens, rates):
        p = rng.integers(0, 4, length)
        hit = rng.random(length) < rate
        t = np.where(hit, (p + rng.integers(1, 4, length)) % 4, p)
        pats.append(np.frombuffer(b"ACGT", np.uint8)[p].tobytes())
        txts.append(np.frombuffer(b"ACGT", np.uint8)[t].tobytes())
    return pats, txts


def _device(pats, txts):
    ps = workloads.from_lists("replay", pats, txts)
    return api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cuda")


def _wfa_outs(torch, b):
    return (torch.full((b.n,), -7, dtype=torch.int32, device="cuda"),
            torch.full((b.n,), -7, dtype=torch.int32, device="cuda"),
            torch.zeros(max(b.out_bytes, 1), dtype=torch.uint8, device="cuda"))


def _check_wfa(b, outs, want, label):
    sc, ln, cg = (t.cpu().numpy() for t in outs)
    assert np.array_equal(sc, want.score), label
    ends = b.out_off.cpu().numpy() + b.a_len.cpu().numpy().astype(np.int64) + b.b_len.cpu().numpy()
    for i, c in enumerate(want.cigars):
        assert int(ln[i]) == len(c) and cg[ends[i] - len(c):ends[i]].tobytes() == c, (label, i)


# mixed reads on lanes and warps; long pairs, some estimated past 256 edits (blocks on a second stream) and
# some below that the warps leave to blocks
MIXED = (np.random.default_rng(1).integers(100, 260, 400), np.random.default_rng(2).uniform(0.0, 0.2, 400), 64)
LONG = (np.random.default_rng(3).integers(900, 2600, 40), np.random.default_rng(4).uniform(0.01, 0.35, 40), 1024)


@pytest.mark.parametrize("trace", [True, False])
@pytest.mark.parametrize("shape", [MIXED, LONG], ids=["mixed", "long"])
def test_learned_wfa_device_calls(shape, trace):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    lens, rates, smax = shape
    sets = [_substituted(seed, lens, rates) for seed in (11, 12)]
    want = [oracle.wfa_batch(p, t, smax=smax, with_cigar=True, max_smax=4096) for p, t in sets]
    b, other = _device(*sets[0]), _device(*sets[1])
    outs = _wfa_outs(torch, b)
    for call, which in enumerate((0, 0, 1, 0)):
        b.seq.copy_((_device(*sets[0]) if which == 0 else other).seq)
        for t in outs:
            t.fill_(-7 if t.dtype == torch.int32 else 0)
        torch.cuda.synchronize()
        api.wfa_device(b, smax, trace, *outs, learned=True)
        if trace:
            _check_wfa(b, outs, want[which], call)
        else:
            assert np.array_equal(outs[0].cpu().numpy(), want[which].score), call


@pytest.mark.parametrize("shape", [MIXED, (LONG[0][:20], LONG[1][:20] * 0.6, 511)], ids=["mixed", "long"])
def test_learned_wfa_host_calls(shape):
    assert cost_model.load_default()
    lens, rates, smax = shape
    for cigar in (True, False):
        for call, seed in enumerate((21, 21, 22)):
            pats, txts = _substituted(seed, lens, rates)
            ps = workloads.from_lists("replay", pats, txts)
            want = oracle.wfa_batch(pats, txts, smax=smax, with_cigar=True)
            got = api.align_batch_packed(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, smax=smax,
                                         with_cigar=cigar, learned=True)
            assert got.status == api.Status.ok, got.error
            assert np.array_equal(got.res["score"], want.score), (cigar, call)
            if cigar:
                assert all(got.cigar(i) == c for i, c in enumerate(want.cigars)), call


def test_learned_calls_that_share_all_but_one_buffer():
    """One query set against two target sets, and outputs of their own: the
    second batch has its own results, written where it asked."""
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    lens, rates, smax = MIXED
    pats, first = _substituted(31, lens, rates)
    rng = np.random.default_rng(32)
    second = [bytes(c if rng.random() > 0.1 else b"ACGT"[rng.integers(0, 4)] for c in t) for t in first]
    both = _device(pats + pats, first + second)
    n = len(pats)
    want = [oracle.wfa_batch(pats, t, smax=smax, with_cigar=True) for t in (first, second)]
    a_off, a_len, out_off = both.a_off[:n].clone(), both.a_len[:n].clone(), both.out_off[:n].clone()
    sides = [(both.b_off[k * n:(k + 1) * n].clone(), both.b_len[k * n:(k + 1) * n].clone()) for k in (0, 1)]

    class View:
        pass

    def view(k):
        v = View()
        v.n, v.a_off, v.a_len, v.out_off = n, a_off, a_len, out_off
        v.b_off, v.b_len = sides[k]
        v.out_bytes = int(both.out_bytes)
        v.c = api.DeviceBatch(both.seq.data_ptr(), both.seq.numel(), a_off.data_ptr(), a_len.data_ptr(),
                              v.b_off.data_ptr(), v.b_len.data_ptr(), out_off.data_ptr(), n, 0)
        return v

    b0, b1 = view(0), view(1)
    outs = _wfa_outs(torch, b0)
    for call in range(3):
        api.wfa_device(b0, smax, True, *outs, learned=True)
        _check_wfa(b0, outs, want[0], call)
    for call in range(3):
        for t in outs:
            t.fill_(-7 if t.dtype == torch.int32 else 0)
        torch.cuda.synchronize()
        api.wfa_device(b1, smax, True, *outs, learned=True)
        _check_wfa(b1, outs, want[1], ("second targets", call))
    fresh = torch.full_like(outs[1], -7)
    kept = outs[1].clone().fill_(-9)
    outs[1].copy_(kept)
    torch.cuda.synchronize()
    api.wfa_device(b1, smax, True, outs[0], fresh, outs[2], learned=True)
    _check_wfa(b1, (outs[0], fresh, outs[2]), want[1], "fresh lengths")
    assert torch.equal(outs[1], kept)


def test_sw_host_calls():
    lens = np.random.default_rng(5).integers(80, 900, 300)
    rates = np.random.default_rng(6).uniform(0.0, 0.2, 300)
    for cigar in (True, False):
        for call, seed in enumerate((41, 41, 42)):
            pats, txts = _substituted(seed, lens, rates)
            ps = workloads.from_lists("replay", txts, pats)
            want = oracle.sw_batch(txts, pats, scoring=SCORING, with_cigar=True)
            got = api.align_sw_batch_packed(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len,
                                            scoring=SCORING, with_cigar=cigar)
            assert got.status == api.Status.ok, got.error
            assert np.array_equal(got.res["score"], want.score), (cigar, call)
            if cigar:
                for f in POS:
                    assert np.array_equal(got.res[f], getattr(want, f)), (call, f)
                assert all(got.cigar(i) == c for i, c in enumerate(want.cigars)), call
