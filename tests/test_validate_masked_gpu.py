"""The device result checks on pairs without a CIGAR: a pair whose score says so (a
caller may have set it) has flags 0 whatever its length and cells hold."""
import numpy as np
import pytest

from genoaligner_gb300 import api, workloads

pytestmark = pytest.mark.gpu

SCORING = (2, -3, 3, 1)


@pytest.mark.parametrize("kind", ["wfa", "sw"])
def test_masked_pairs(kind):
    torch = pytest.importorskip("torch")
    ps = workloads.wfa_mixed(n=500, seed=71) if kind == "wfa" else workloads.sw_uneven_200k(n=500, seed=72)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cuda")
    score, length = (torch.empty(b.n, dtype=torch.int32, device="cuda") for _ in range(2))
    pos = torch.empty(4 * b.n, dtype=torch.int32, device="cuda")
    cigar = torch.zeros(b.out_bytes, dtype=torch.uint8, device="cuda")
    flags, again = (torch.full((b.n,), 9, dtype=torch.uint8, device="cuda") for _ in range(2))
    if kind == "wfa":
        api.wfa_device(b, 64, True, score, length, cigar)
        check = lambda f: api.wfa_validate_device(b, score, length, cigar, f)        # noqa: E731
    else:
        api.sw_device(b, SCORING, True, score, pos, length, cigar)
        check = lambda f: api.sw_validate_device(b, SCORING, score, pos, length, cigar, f)        # noqa: E731
    check(flags)
    torch.cuda.synchronize()
    assert int((flags == 3).sum()) > 400
    rng = np.random.default_rng(73)
    out = torch.from_numpy(rng.permutation(b.n)[:200]).cuda()
    score[out] = -1
    length[out[:150]] = torch.from_numpy(rng.integers(1, 1 << 30, 150).astype(np.int32)).cuda()
    pos.view(-1, 4)[out[100:]] = -1
    torch.cuda.synchronize()
    check(again)
    torch.cuda.synchronize()
    want = flags.clone()
    want[out] = 0
    assert torch.equal(again, want)
