"""Smith-Waterman items that a whole block computes: batches of few pairs around the
bands' edges, fewer bands than warps and more, shapes where one row block or one band
is all there is, ties between bands, every block size, each list (16-bit, 32-bit short
and long shape) and both entries; and a batch whose leading items only are such."""
import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, workloads
from helpers import assert_sw_equal, packed, sw_gpu

pytestmark = pytest.mark.gpu

SCORING = (2, -3, 5, 2)


def _pairs(m, n, seed, impure):
    """Three pairs: related, a period of two letters (equal bests in many bands), unrelated."""
    rng = np.random.default_rng(seed)
    ts, ps = [], []
    for kind in range(3):
        p = np.tile(np.frombuffer(b"AC", np.uint8), n)[:n].copy() if kind == 1 else workloads.random_bases(rng, n)
        t = workloads.random_bases(rng, m)
        if kind == 0:
            q = workloads.mutate_runs(rng, p, 0.08, (0.6, 0.2, 0.2), 0.3)[: m - m // 8]
            t[m // 8: m // 8 + q.shape[0]] = q
        elif kind == 1:
            t[::3] = ord("A")
        if impure:
            p[n // 2] = ord("r")
        ts.append(t.tobytes())
        ps.append(p.tobytes())
    return ts, ps


SHAPES = [(300, 300), (511, 513), (640, 1025), (1031, 127), (1000, 128), (600, 129), (65, 1100), (2, 40000),
          (70000, 1), (33, 4200), (1500, 2100), (4600, 4150)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("with_cigar", [True, False])
def test_few_pairs_match_oracle(shape, with_cigar):
    for impure in (False, True):
        ts, ps = _pairs(*shape, 40 + shape[0], impure)
        want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=with_cigar)
        if not with_cigar and want.status != "ok":
            continue                                   # wider than the score-only entry takes
        for k in (3, 1):
            sub = oracle.sw_batch(ts[:k], ps[:k], scoring=SCORING, with_cigar=with_cigar)
            assert_sw_equal(sw_gpu(ts[:k], ps[:k], scoring=SCORING, with_cigar=with_cigar), sub,
                            f"{shape}, {k} pairs, impure {impure}")


@pytest.mark.parametrize("shape", [(1100, 1100), (3000, 2100), (1300, 4500)])
@pytest.mark.parametrize("entry", ["host", "device"])
def test_settings_agree(shape, entry):
    """The 32-bit shapes and no whole-block items at all give the same alignments, from
    the plan on the device and from the one read back."""
    torch = pytest.importorskip("torch")
    ts, ps = _pairs(*shape, 7, False)
    want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=True)
    before = api.tune_get()
    try:
        for setting in (dict(), dict(sw_pack16=0), dict(sw_pack16=0, sw_long_log2=20), dict(sw_coop_log2=40),
                        dict(sw_window=4), dict(sw_pack16=0, sw_long_log2=20, sw_coop_log2=16)):
            api.tune_set(**{**before, **setting})
            if entry == "host":
                assert_sw_equal(sw_gpu(ts, ps, scoring=SCORING), want, f"{shape}, {setting}")
                continue
            q = packed(ts, ps)
            batch = api.DeviceBatchT(q.a_buf, q.a_off, q.a_len, q.b_buf, q.b_off, q.b_len)
            n = len(ts)
            score, pos, length = (torch.zeros(k * n, dtype=torch.int32, device="cuda") for k in (1, 4, 1))
            cigar = torch.zeros(batch.out_bytes, dtype=torch.uint8, device="cuda")
            api.sw_device(batch, SCORING, True, score, pos, length, cigar)
            host = sw_gpu(ts, ps, scoring=SCORING)
            assert np.array_equal(score.cpu().numpy(), want.score)
            got, ends = cigar.cpu().numpy(), (batch.out_off + batch.a_len + batch.b_len).cpu().numpy()
            for k in range(n):
                ln = int(length[k])
                assert got[int(ends[k]) - ln: int(ends[k])].tobytes() == host.cigar(k), (shape, setting, k)
    finally:
        api.tune_set(**before)


@pytest.mark.parametrize("with_cigar", [True, False])
def test_leading_items_only(with_cigar):
    rng = np.random.default_rng(5)
    ts, ps = [], []
    for k in range(3040):
        m, n = (2000 + k, 1600 + 3 * k) if k < 40 else (int(rng.integers(1, 120)), int(rng.integers(1, 90)))
        p = workloads.random_bases(rng, n)
        t = np.concatenate([workloads.random_bases(rng, max(0, m - n) // 2),
                            workloads.mutate_runs(rng, p, 0.1, (0.6, 0.2, 0.2))])[:m]
        if k % 9 == 0:
            p[0] = ord("x")
        ts.append(t.tobytes())
        ps.append(p.tobytes())
    order = rng.permutation(len(ts))
    ts, ps = [ts[k] for k in order], [ps[k] for k in order]
    if not with_cigar:
        ps = [p[:1500] for p in ps]
    want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=with_cigar)
    assert_sw_equal(sw_gpu(ts, ps, scoring=SCORING, with_cigar=with_cigar), want, "leading items")


@pytest.mark.parametrize("n", [1, 31, 1025, 4095, 4096, 4097])
def test_plan_by_one_block_and_by_many(n):
    """Every list non-empty, at the sizes around what one block plans."""
    rng = np.random.default_rng(n)
    ts, ps = [], []
    for k in range(n):
        p = workloads.random_bases(rng, int(rng.integers(0, 70)))
        t = np.concatenate([workloads.random_bases(rng, int(rng.integers(0, 9))), workloads.mutate_runs(rng, p, 0.1, (0.6, 0.2, 0.2))])
        if k % 3 == 1 and p.shape[0]:
            p[-1] = ord("y")
        if k % 400 == 30:
            p, t = workloads.random_bases(rng, 1100), workloads.random_bases(rng, 1000 + k % 7)
            if k % 800 == 30:
                p[3] = ord("-")
        ts.append(t.tobytes())
        ps.append(p.tobytes())
    before = api.tune_get()
    try:
        api.tune_set(**{**before, "sw_long_log2": 20})
        for with_cigar in (True, False):
            want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=with_cigar)
            assert_sw_equal(sw_gpu(ts, ps, scoring=SCORING, with_cigar=with_cigar), want, f"{n} pairs, {with_cigar}")
    finally:
        api.tune_set(**before)


def test_device_entry_lists_side_by_side_after_the_arena_grew():
    """Long pairs of both widths (two streams), three times the size of the call before:
    the plan is made again in the grown arena and sized again."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(8)
    for n in (2, 30, 90):
        ts, ps = [], []
        for k in range(n):
            p = workloads.random_bases(rng, int(rng.integers(300, 1500)))
            t = np.concatenate([workloads.mutate_runs(rng, p, 0.1, (0.6, 0.2, 0.2)),
                                workloads.random_bases(rng, int(rng.integers(0, 400)))])
            if k % 2:
                p[p.shape[0] // 2] = ord("q")
            ts.append(t.tobytes())
            ps.append(p.tobytes())
        want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=True)
        q = packed(ts, ps)
        batch = api.DeviceBatchT(q.a_buf, q.a_off, q.a_len, q.b_buf, q.b_off, q.b_len)
        before = api.tune_get()
        try:
            api.tune_set(**{**before, "sw_long_log2": 20})
            score, pos, length = (torch.zeros(k * n, dtype=torch.int32, device="cuda") for k in (1, 4, 1))
            cigar = torch.zeros(batch.out_bytes, dtype=torch.uint8, device="cuda")
            for limit in (-1, 1 << 26, 1 << 26, 1 << 26):           # as it is, then captured and replayed
                score.zero_()
                cigar.zero_()
                api.sw_device(batch, SCORING, True, score, pos, length, cigar, trace_cell_limit=limit)
                assert np.array_equal(score.cpu().numpy(), want.score)
                got, ends = cigar.cpu().numpy(), (batch.out_off + batch.a_len + batch.b_len).cpu().numpy()
                for k in range(n):
                    assert got[int(ends[k]) - int(length[k]): int(ends[k])].tobytes() == want.cigars[k], (n, limit, k)
        finally:
            api.tune_set(**before)


@pytest.mark.parametrize("rows", [65535, 65536, 70000])
def test_texts_past_16_bit_rows(rows):
    """The alignment ends in the last rows of a text that 16 bits just hold or do not."""
    rng = np.random.default_rng(rows)
    p = workloads.random_bases(rng, 60)
    t = workloads.random_bases(rng, rows)
    t[-70:-10] = p
    t2 = workloads.random_bases(rng, 900)
    ts, ps = [t.tobytes(), t2.tobytes()], [p.tobytes(), t2[100:700].tobytes()]
    for with_cigar in (True, False):
        want = oracle.sw_batch(ts, ps, scoring=SCORING, with_cigar=with_cigar)
        assert_sw_equal(sw_gpu(ts, ps, scoring=SCORING, with_cigar=with_cigar), want, f"{rows} rows, {with_cigar}")
