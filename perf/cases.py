"""What is timed: the calls that programs make into this library, over the range they make them.

A case is a dict of plain values.  ``op`` names the kind of call:

* ``wfa``: bounded edit distance of n (pattern, text) pairs, ``align_batch`` on host buffers (``entry`` "host")
  or ``wfa_device`` on sequences already in device memory ("device");
* ``sw``: affine Smith-Waterman of n (text, pattern) pairs, ``align_sw_batch`` or ``sw_device``;
* ``fit``: one batch of the cost model's training, its loss and the gradient of every parameter.

Sequences are seeded random DNA: a source of ``len_lo`` to ``len_hi`` bases (lengths spread over their logarithm)
and a copy with substitutions, insertions and deletions at a rate drawn per pair from ``err_lo`` to ``err_hi``
(``mixture``: 70 % of the pairs at 0-2 %, 25 % at 2-10 %, 5 % at 10-30 %; ``runs``: indels of geometric length).
Smith-Waterman texts carry ``flank`` random bases at most on either side of the copy; ``shared`` pairs have one
pattern, the same buffer in every request; ``impure`` is the share of copies that hold some N.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from genoaligner_gb300 import api, cost_model

DEVICE = "cuda"
SCORING = (2, -3, 3, 1)


def _wfa(name, entry, n, lo, hi, err, smax, **more):
    return {"name": name, "op": "wfa", "entry": entry, "n": n, "len_lo": lo, "len_hi": hi, "err_lo": err[0],
            "err_hi": err[1], "mixture": False, "runs": False, "impure": 0.0, "smax": smax, "cigar": True,
            "learned": False, **more}


def _sw(name, entry, n, lo, hi, flank, err, **more):
    return {"name": name, "op": "sw", "entry": entry, "n": n, "len_lo": lo, "len_hi": hi, "flank": flank,
            "err_lo": err[0], "err_hi": err[1], "shared": False, "impure": 0.0, "cigar": True, **more}


def listed():
    return [
        # one gene against one reference, as an interactive program or a service aligns it: latency
        _sw("sw_one_pair", "host", 1, 1000, 1000, 100, (0.05, 0.05)),
        # a handful of reads checked against their candidate positions: latency
        _wfa("wfa_48_reads", "host", 48, 140, 160, (0.0, 0.05), 64),
        # a chunk of short reads from host buffers, scores and CIGARs
        _wfa("wfa_10k_reads", "host", 10_000, 150, 150, (0.02, 0.02), 64),
        # a whole read set of mixed divergence in device memory, routed by the cost model
        _wfa("wfa_1m_mixed", "device", 1_000_000, 150, 250, (0.0, 0.3), 64, mixture=True, learned=True),
        # distances alone of 2 kb amplicons, by the plain kernels
        _wfa("wfa_20k_score", "device", 20_000, 1800, 2200, (0.0, 0.1), 256, cigar=False),
        # long reads of 1-10 kb, divergent, with CIGARs, routed by the cost model
        _wfa("wfa_2k_long", "device", 2000, 1000, 10_000, (0.01, 0.15), 2048, runs=True, learned=True),
        # scores of some hundred pairs up to 1 kb, as a clustering step asks for them
        _sw("sw_600_score", "host", 600, 200, 1000, 100, (0.0, 0.2), cigar=False),
        # thousands of records of one gene against one reference, some with ambiguous bases
        _sw("sw_3558_gene", "host", 3558, 1137, 1137, 50, (0.0, 0.1), shared=True, impure=0.1),
        # a large batch of uneven pairs in device memory, with CIGARs
        _sw("sw_200k_uneven", "device", 200_000, 50, 1000, 500, (0.05, 0.05)),
        # the same batch from host buffers and back to them
        _sw("sw_200k_host", "host", 200_000, 50, 1000, 500, (0.05, 0.05)),
        # long pairs, whose tables outgrow 16 bits and one warp
        _sw("sw_1k_long", "device", 1024, 2000, 30_000, 5000, (0.1, 0.1)),
        # one training batch of the cost model (forward, backward)
        {"name": "fit_8192", "op": "fit", "n": 8192},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["wfa_host", "wfa_device", "wfa_long", "sw_host", "sw_device", "sw_long", "fit"])
    if kind == "wfa_host":
        lo = _log_uniform(rng, 60, 300)
        top = rng.choice([0.02, 0.05, 0.1])
        case = _wfa("", "host", _log_uniform(rng, 1, 300_000), lo, int(lo * rng.uniform(1.0, 2.0)), (0.0, top),
                    rng.choice([31, 64, 100]), cigar=rng.random() < 0.7, impure=rng.choice([0.0, 0.05]))
    elif kind == "wfa_device":
        lo = rng.randint(100, 200)
        case = _wfa("", "device", _log_uniform(rng, 5000, 1_000_000), lo, int(lo * rng.uniform(1.0, 1.6)),
                    (0.0, 0.3), rng.choice([48, 64]), mixture=True, learned=rng.random() < 0.5,
                    cigar=rng.random() < 0.7)
    elif kind == "wfa_long":
        lo = _log_uniform(rng, 1000, 3000)
        case = _wfa("", "device", _log_uniform(rng, 100, 2000), lo, int(lo * rng.uniform(1.0, 3.3)), (0.01, 0.12),
                    rng.choice([256, 511, 1024, 2048]), runs=True, learned=rng.random() < 0.5,
                    cigar=rng.random() < 0.5)
    elif kind == "sw_host":
        lo = _log_uniform(rng, 50, 1000)
        hi = int(lo * rng.uniform(1.0, 1.5))
        case = _sw("", "host", _log_uniform(rng, 1, 20_000), lo, hi, rng.randint(0, 300), (0.0, rng.choice([0.05, 0.2])),
                   shared=rng.random() < 0.3, impure=rng.choice([0.0, 0.1]), cigar=rng.random() < 0.7)
    elif kind == "sw_device":
        lo = _log_uniform(rng, 50, 300)
        case = _sw("", "device", _log_uniform(rng, 2000, 200_000), lo, int(lo * rng.uniform(1.0, 3.3)),
                   rng.randint(0, 500), (0.02, 0.08), cigar=rng.random() < 0.7)
    elif kind == "sw_long":
        lo = _log_uniform(rng, 2000, 8000)
        case = _sw("", "device", _log_uniform(rng, 32, 1024), lo, int(lo * rng.uniform(1.0, 1.8)),
                   rng.randint(0, 5000), (0.05, 0.15))
    else:
        case = {"name": "", "op": "fit", "n": _log_uniform(rng, 500, 8192)}
    del case["name"]
    return case


# ----------------------------------------------------------------- inputs --
class _Random:
    """Draws on the device from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(seed)

    def uniform(self, n, lo=0.0, hi=1.0):
        return torch.rand(n, generator=self.g, device=DEVICE) * (hi - lo) + lo

    def integers(self, n, lo, hi, dtype=torch.int64):
        return torch.randint(lo, hi, (n,), generator=self.g, device=DEVICE, dtype=dtype)


def _starts(lens):
    return torch.cumsum(lens, 0) - lens


def _place(dst, dst_start, src, lens):
    """Segment s of src (lens[s] values, one after the other) to dst[dst_start[s]:]."""
    at = torch.repeat_interleave(dst_start - _starts(lens), lens)
    at += torch.arange(at.numel(), device=DEVICE)
    dst[at] = src


def _mutate(r, src, lens, rate, mix, runs):
    """Copies of the segments of src (codes 0-3) with errors; (codes, lengths)."""
    total = src.numel()
    event = (r.uniform(total) < torch.repeat_interleave(rate, lens)).nonzero().squeeze(1)
    kind = r.uniform(event.numel())
    sub = event[kind < mix[0]]
    ins = event[(kind >= mix[0]) & (kind < mix[0] + mix[1])]
    dele = event[kind >= mix[0] + mix[1]]

    def run_lengths(count):
        if not runs:
            return torch.ones(count, dtype=torch.int64, device=DEVICE)
        return 1 + torch.floor(torch.log2(1.0 / r.uniform(count).clamp_min(1e-6))).to(torch.int64)

    vals = src.clone()
    vals[sub] = (vals[sub] + r.integers(sub.numel(), 1, 4, torch.uint8)) % 4
    reps = torch.ones(total, dtype=torch.int64, device=DEVICE)
    reps[ins] += run_lengths(ins.numel())
    ends = torch.cumsum(lens, 0)
    stop = torch.minimum(dele + run_lengths(dele.numel()), ends[torch.searchsorted(ends, dele, right=True)])
    gone = torch.zeros(total + 1, dtype=torch.int32, device=DEVICE)
    one = torch.ones_like(dele, dtype=torch.int32)
    gone.index_add_(0, dele, one)
    gone.index_add_(0, stop, -one)
    reps[torch.cumsum(gone, 0)[:total] > 0] = 0
    out = torch.repeat_interleave(vals, reps)
    first = torch.zeros(out.numel(), dtype=torch.bool, device=DEVICE)
    first[_starts(reps)[reps > 0]] = True
    out = torch.where(first, out, r.integers(out.numel(), 0, 4, torch.uint8))
    upto = torch.cumsum(reps, 0)[ends - 1]
    return out, torch.diff(upto, prepend=upto.new_zeros(1))


def _letters(codes):
    return torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEVICE)[codes.long()]


def _pairs(case, seed):
    """(source letters, lengths, copy letters, lengths): side by side in pair order, on the device."""
    r = _Random(seed)
    n = case["n"]
    if case.get("shared"):
        one = r.integers(case["len_lo"], 0, 4, torch.uint8)
        lens = torch.full((n,), one.numel(), device=DEVICE)
        src = one.repeat(n)
    else:
        lens = torch.exp(r.uniform(n, math.log(case["len_lo"]), math.log(case["len_hi"]))).round().to(torch.int64)
        src = r.integers(int(lens.sum()), 0, 4, torch.uint8)
    if case.get("mixture"):
        part = r.uniform(n)
        lo = torch.where(part < 0.7, 0.0, torch.where(part < 0.95, 0.02, 0.1))
        hi = torch.where(part < 0.7, 0.02, torch.where(part < 0.95, 0.1, 0.3))
    else:
        lo, hi = torch.tensor(case["err_lo"], device=DEVICE), torch.tensor(case["err_hi"], device=DEVICE)
    rate = lo + (hi - lo) * r.uniform(n)
    mix = (1 / 3, 1 / 3) if case["op"] == "wfa" else (0.6, 0.2)
    copy, copy_len = _mutate(r, src, lens, rate, mix, case.get("runs", False))
    if case.get("flank"):
        left, right = (r.integers(n, 0, case["flank"] + 1) for _ in range(2))
        text_len = left + copy_len + right
        text = r.integers(int(text_len.sum()), 0, 4, torch.uint8)
        _place(text, _starts(text_len) + left, copy, copy_len)
        copy, copy_len = text, text_len
    copy = _letters(copy)
    if case["impure"]:
        marked = torch.repeat_interleave(r.uniform(n) < case["impure"], copy_len)
        copy[marked & (r.uniform(copy.numel()) < 0.01)] = ord("N")
    return _letters(src), lens, copy, copy_len


def _device_batch(a, a_len, b, b_len):
    ra, rb = (a_len + 31) // 32 * 32, (b_len + 31) // 32 * 32
    a_off = _starts(ra + rb)
    arena = torch.zeros(int((ra + rb).sum()) + 64, dtype=torch.uint8, device=DEVICE)
    _place(arena, a_off, a, a_len)
    _place(arena, a_off + ra, b, b_len)
    return api.DeviceBatchT.from_device_arena(arena, a_off.cpu().numpy(), a_len.cpu().numpy(),
                                              (a_off + ra).cpu().numpy(), b_len.cpu().numpy())


def _mean_len(case):
    lo, hi = case["len_lo"], case["len_hi"]
    return (hi - lo) / math.log(hi / lo) if hi > lo else lo


def _cigar_room(case):
    """CIGAR bytes held for a batch: both sides' letters at the mean sizes and a margin, whatever was drawn."""
    flank = case.get("flank", 0)
    return int(1.1 * case["n"] * (2 * _mean_len(case) + flank) + 8 * math.sqrt(case["n"]) * (case["len_hi"] + flank)) + 64


def _host_side(buf, lens):
    return buf.cpu().numpy(), _starts(lens).cpu().numpy(), lens.to(torch.int32).cpu().numpy()


def prepare(case, seed):
    if case["op"] == "fit":
        cost_model.load_default()
        r = _Random(seed)
        n = case["n"]
        feat = torch.cat([r.integers(64 * n, -6, 7).view(n, 64) / 8.0, r.uniform(2 * n, 0.55, 1.0).view(n, 2)], 1)
        dist = torch.exp2(r.uniform(n, 0.0, 6.0)).floor()
        target = torch.stack([torch.log2(dist + 1), torch.log2((dist + 1) ** 2 + 1)], 1)
        return {"case": case, "feat": feat.contiguous(), "target": target.contiguous()}
    if case.get("learned"):
        cost_model.load_default()
    src, src_len, copy, copy_len = _pairs(case, seed)
    # edit distance: pattern = source, text = copy; Smith-Waterman: text = copy, pattern = source
    a, a_len, b, b_len = (src, src_len, copy, copy_len) if case["op"] == "wfa" else (copy, copy_len, src, src_len)
    n = case["n"]
    state = {"case": case}
    if case["entry"] == "host":
        sa, sb = _host_side(a, a_len), _host_side(b, b_len)
        if case.get("shared"):
            sb = (sb[0][:case["len_lo"]].copy(), np.zeros_like(sb[1]), sb[2])
        make, dt = (api.make_requests, api.RES_DT) if case["op"] == "wfa" else (api.make_sw_requests, api.SWRES_DT)
        extra = {"smax": case["smax"]} if case["op"] == "wfa" else {"scoring": SCORING}
        state.update(sides=sa + sb, reqs=make(*sa, *sb, with_cigar=case["cigar"], **extra), res=np.zeros(n, dt),
                     cigar=np.zeros(_cigar_room(case), np.uint8))
    else:
        batch = _device_batch(a, a_len, b, b_len)
        out = {"score": torch.zeros(n, dtype=torch.int32, device=DEVICE)}
        if case["op"] == "sw":
            out["pos"] = torch.zeros(4 * n, dtype=torch.int32, device=DEVICE)
        if case["cigar"]:
            out["len"] = torch.zeros(n, dtype=torch.int32, device=DEVICE)
            out["cigar"] = torch.zeros(_cigar_room(case), dtype=torch.uint8, device=DEVICE)
            assert out["cigar"].numel() >= batch.out_bytes
        state.update(batch=batch, out=out)
    return state


# ------------------------------------------------------------------- calls --
def run(state):
    case = state["case"]
    if case["op"] == "fit":
        grad, loss = api.mlp_gradient(state["feat"], state["target"])
        return {"grad": grad, "loss": loss}
    if case["entry"] == "host":
        held = {"_reqs": state["reqs"], "_res": state["res"], "_cig": state["cigar"]}
        if case["op"] == "wfa":
            api.align_batch_packed(*state["sides"], smax=case["smax"], with_cigar=case["cigar"], **held)
        else:
            api.align_sw_batch_packed(*state["sides"], scoring=SCORING, with_cigar=case["cigar"], **held)
        out = {"res": state["res"].view(np.int32)}
        if case["cigar"]:
            out["cigar"] = state["cigar"]
        return out
    out = state["out"]
    if case["op"] == "wfa":
        api.wfa_device(state["batch"], case["smax"], case["cigar"], out["score"], out.get("len"), out.get("cigar"),
                       learned=case["learned"])
    else:
        api.sw_device(state["batch"], SCORING, case["cigar"], out["score"], out["pos"], out.get("len"),
                      out.get("cigar"))
    return out


# --------------------------------------------------------------- the least --
def work(case):
    """Bytes in and out of one pass at the mean sizes, and the integer (or fp32) operations of its recurrence."""
    n = case["n"]
    if case["op"] == "fit":
        params = 66 * 128 + 128 * 128 + 128 * 2
        return {"bytes": n * 68 * 4 + 4 * (params + 258), "flops": 6 * params * n}
    lo, hi, mean = case["len_lo"], case["len_hi"], _mean_len(case)
    rate = 0.7 * 0.01 + 0.25 * 0.06 + 0.05 * 0.2 if case.get("mixture") else (case["err_lo"] + case["err_hi"]) / 2
    text = mean + case.get("flank", 0)
    moved = mean + text + 24 + (40 if case["entry"] == "host" else 8)
    if case["cigar"]:
        moved += mean * (1 + rate)
    if case["op"] == "wfa":
        dist = min(case["smax"], mean * rate * (1.5 if case["runs"] else 1.0))
        return {"bytes": n * moved, "flops": n * 8 * (dist + 1) ** 2}
    square = (hi * hi - lo * lo) / (2 * math.log(hi / lo)) if hi > lo else lo * lo
    return {"bytes": n * moved, "flops": n * 6 * (square + mean * case["flank"])}


def exact(case, seed):
    """The gradient and loss of a training batch in 64 bits, with the weights rounded to bfloat16 as the network's
    forward pass holds them; the alignments are whole numbers and have none."""
    if case["op"] != "fit":
        return None
    state = prepare(case, seed)
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genoaligner_gb300", "models",
                        "wfa_cost_v1.npz")
    p = torch.from_numpy(np.load(path)["params"]).to(torch.bfloat16).double()
    w1, b1, w2, b2, w3, b3 = (q.to(DEVICE) for q in torch.split(p, [128 * 66, 128, 128 * 128, 128, 2 * 128, 2]))
    w1, w2, w3 = w1.view(128, 66), w2.view(128, 128), w3.view(2, 128)
    x, t = state["feat"].double(), state["target"].double()
    h1 = torch.relu(x @ w1.T + b1)
    h2 = torch.relu(h1 @ w2.T + b2)
    e = h2 @ w3.T + b3 - t
    d3 = 2 * e / x.shape[0]
    d2 = (d3 @ w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = torch.cat([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), (d3.T @ h2).reshape(-1),
                      d3.sum(0)])
    return {"grad": grad.cpu().numpy(), "loss": float((e * e).sum())}
