"""The passes of plain WFA batches (on a runtime that records, no GPU): above smax 511 the
warps search 255 edits and blocks take the pairs left; where more could be left than
blocks are quick with, a second warp pass is launched for that case."""
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, workloads


@pytest.mark.parametrize("n,smax,blocks,second", [(100, 511, 0, 0), (100, 512, 1, 0), (500, 1024, 1, 0),
                                                  (5000, 511, 0, 0), (5000, 512, 1, 1), (5000, 700, 1, 1),
                                                  (5000, 701, 1, 1), (5000, 2048, 1, 1)])
@pytest.mark.parametrize("trace", [True, False])
def test_passes(rt, n, smax, blocks, second, trace):
    torch = pytest.importorskip("torch")
    ps = workloads.wfa_mixed(n=n, seed=1)
    b = api.DeviceBatchT(ps.a_buf, ps.a_off, ps.a_len, ps.b_buf, ps.b_off, ps.b_len, device="cpu")
    rt.clear()
    api.wfa_device(b, smax, trace, torch.zeros(n, dtype=torch.int32), torch.zeros(n, dtype=torch.int32),
                   torch.zeros(b.out_bytes, dtype=torch.uint8))
    kernel = f"wfa_kernelILb{int(trace)}ELi"            # <trace, pass>
    assert rt.count(kernel + ("1E" if second else "0E")) == 1
    assert (rt.count("wfa_block_kernel"), rt.count(kernel + "2E")) == (blocks, second)
