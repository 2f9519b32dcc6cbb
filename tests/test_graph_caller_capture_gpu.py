"""WFA device calls recorded into a graph that the caller captures: a warmed shape is
recorded and replays on changed sequences, a second call (plain) is recorded too or
(learned, another shape) refused and leaves the capture as it was, and calls after the
capture work as before."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, cost_model, workloads

pytestmark = pytest.mark.gpu


def _batch(torch, seed, n=300):
    rng = np.random.default_rng(7)
    lens = rng.integers(100, 260, n)
    rng = np.random.default_rng(seed)
    pats, txts = [], []
    for length in lens:
        p = workloads.random_bases(rng, int(length))
        t = np.where(rng.random(int(length)) < 0.1, workloads.random_bases(rng, int(length)), p)
        pats.append(p.tobytes())
        txts.append(t.tobytes())
    ps = workloads.from_lists("capture", pats, txts)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cuda")
    return b, oracle.wfa_batch(pats, txts, smax=64, with_cigar=True)


def _outs(torch, b):
    return (torch.full((b.n,), -7, dtype=torch.int32, device="cuda"),
            torch.full((b.n,), -7, dtype=torch.int32, device="cuda"),
            torch.zeros(b.out_bytes, dtype=torch.uint8, device="cuda"))


def _check(b, outs, want, label):
    sc, ln, cg = (t.cpu().numpy() for t in outs)
    assert np.array_equal(sc, want.score), label
    ends = b.out_off.cpu().numpy() + b.a_len.cpu().numpy().astype(np.int64) + b.b_len.cpu().numpy()
    for i, c in enumerate(want.cigars):
        assert int(ln[i]) == len(c) and cg[ends[i] - len(c):ends[i]].tobytes() == c, (label, i)


@pytest.mark.parametrize("learned", [True, False])
@pytest.mark.parametrize("warm_calls", [1, 2])
def test_capture_of_a_warmed_shape(learned, warm_calls):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    b, want = _batch(torch, 1)
    other, other_want = _batch(torch, 2)
    outs, second = _outs(torch, b), _outs(torch, b)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(warm_calls):
        api.wfa_device(b, 64, True, *outs, stream=s.cuda_stream, learned=learned)
    s.synchronize()
    _check(b, outs, want, "warm")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        if learned:
            with pytest.raises(RuntimeError):
                api.wfa_device(b, 64, True, *second, stream=s.cuda_stream, learned=True)
        else:
            api.wfa_device(b, 64, True, *second, stream=s.cuda_stream)
        api.wfa_device(b, 64, True, *outs, stream=s.cuda_stream, learned=learned)
    for batch, expect in ((b, want), (other, other_want)):
        b.seq.copy_(batch.seq)
        for t in outs:
            t.fill_(-7 if t.dtype == torch.int32 else 0)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        _check(b, outs, expect, "replay")
        if not learned:
            _check(b, second, expect, "replay, first of two")
    for call in range(3):
        for t in outs:
            t.fill_(-7 if t.dtype == torch.int32 else 0)
        torch.cuda.synchronize()
        api.wfa_device(b, 64, True, *outs, stream=s.cuda_stream, learned=learned)
        s.synchronize()
        _check(b, outs, other_want, ("after", call))
