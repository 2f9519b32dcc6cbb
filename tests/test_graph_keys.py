"""Which calls run as CUDA graphs (on a runtime that records, no GPU).  A graph is
replayed only for the call it was captured for: every value the captured launches
hold is in the key.  A call is captured when it repeats the one before; a stream
that cannot be captured takes what that one did, and nothing else."""
import numpy as np
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, cost_model, workloads


def _batch(torch, ps):
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    out = (torch.zeros(b.n, dtype=torch.int32), torch.zeros(b.n, dtype=torch.int32),
           torch.zeros(max(b.out_bytes, 1), dtype=torch.uint8))
    return b, out


def test_equal_learned_calls_replay_one_graph(rt):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    b, out = _batch(torch, workloads.wfa_mixed(n=300, seed=1))
    for call, want in enumerate(((0, 0), (1, 1), (0, 1), (0, 1))):
        rt.clear()
        api.wfa_device(b, 64, True, *out, learned=True)
        assert (rt.count("capture"), rt.count("replay")) == want, call


@pytest.mark.parametrize("changed", ["a_off", "a_len", "b_off", "b_len", "out_off", "out_score", "out_len", "out_cigar",
                                     "seq", "seq_bytes"])
def test_learned_call_with_another_buffer_is_no_replay(rt, changed):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    b, out = _batch(torch, workloads.wfa_mixed(n=300, seed=1))
    for _ in range(3):
        api.wfa_device(b, 64, True, *out, learned=True)
    out = list(out)
    keep = []
    if changed.startswith("out_") and changed != "out_off":
        k = ("out_score", "out_len", "out_cigar").index(changed)
        keep.append(out[k])
        out[k] = out[k].clone()
    elif changed == "seq_bytes":
        b.c.seq_bytes -= 32                       # (every sequence still ends 32 bytes before the end)
    else:
        t = getattr(b, changed)
        keep.append(t)
        t = t.clone()
        keep.append(t)
        setattr(b.c, changed, t.data_ptr())
    rt.clear()
    api.wfa_device(b, 64, True, *out, learned=True)
    assert rt.count("replay") == 0 and rt.count("launch") > 0


def test_host_batches_whose_arenas_share_a_256_byte_step_are_no_replay(rt):
    """Score-only host batches of equal n, arenas 128 bytes apart: each carved
    buffer starts where the other batch's does."""
    assert cost_model.load_default()
    rng = np.random.default_rng(3)

    def call(length):
        a = workloads.random_bases(rng, 32 * 40)
        off = np.arange(40, dtype=np.int64) * 32
        lens = np.full(40, 32, np.int32)
        lens[0] = length                                    # (the second sequence's bytes again)
        got = api.align_batch_packed(a, off, lens, a, off, lens, smax=31, with_cigar=False, learned=True)
        assert got.status == api.Status.ok, got.error

    for _ in range(3):
        call(32)
    for length in (64, 96, 128, 160, 192, 224, 256):
        rt.clear()
        call(length)
        assert rt.count("replay") == 0, length


def test_a_shape_between_two_others_is_not_captured(rt):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    a, b = (_batch(torch, workloads.wfa_mixed(n=n, seed=1)) for n in (300, 200))
    for x in (a, a, b, a, b, a, b):
        api.wfa_device(x[0], 64, True, *x[1], learned=True)
    assert rt.count("capture") == 1                     # a's two in a row


LEGACY = 1                                              # cudaStreamLegacy


@pytest.mark.parametrize("legacy", [True, False])
def test_streams_that_cannot_be_captured(rt, legacy):
    torch = pytest.importorskip("torch")
    assert cost_model.load_default()
    b, out = _batch(torch, workloads.wfa_mixed(n=300, seed=1))
    other, other_out = _batch(torch, workloads.wfa_mixed(n=200, seed=2))
    s = LEGACY if legacy else rt.stream()

    def refused(batch, outs):
        rt.clear()
        if not legacy:
            rt.capturing(s, True)
        try:
            api.wfa_device(batch, 64, True, *outs, stream=s, learned=True)
            return False
        except RuntimeError:
            assert not rt.log()                         # nothing was enqueued
            return True
        finally:
            if not legacy:
                rt.capturing(s, False)

    assert refused(b, out) and refused(b, out)          # a new shape: every time
    api.wfa_device(b, 64, True, *out, learned=True)
    assert not refused(b, out)                          # the shape of the call before
    assert refused(other, other_out)
    for _ in range(2):
        api.wfa_device(b, 64, True, *out, learned=True)
    assert not refused(b, out)
    # a captured shape: replayed, or enqueued into the caller's capture, which takes no graph launch
    assert rt.count("replay") == (1 if legacy else 0) and rt.log()
    api.wfa_device(other, 64, True, *other_out, learned=True)
    assert refused(b, out) and not refused(other, other_out)


def test_plain_calls_take_any_stream(rt):
    torch = pytest.importorskip("torch")
    b, out = _batch(torch, workloads.wfa_mixed(n=300, seed=1))
    s = rt.stream()
    rt.capturing(s, True)
    for stream in (s, LEGACY):
        api.wfa_device(b, 64, True, *out, stream=stream)
    rt.capturing(s, False)
