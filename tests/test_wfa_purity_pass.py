"""Large plain WFA batches set the purity flags in a kernel of their own, small ones
launch one kernel fewer (on a runtime that records, no GPU)."""
import numpy as np
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, workloads


@pytest.mark.parametrize("n", [1, 65535, 65536, 70000])
def test_flags_kernel(rt, n):
    torch = pytest.importorskip("torch")
    a = workloads.random_bases(np.random.default_rng(1), 4 * n)
    off, lens = np.arange(n, dtype=np.int64) * 4, np.full(n, 4, np.int32)
    b = api.DeviceBatchT(a, off, lens, a, off, lens, device="cpu")
    rt.clear()
    api.wfa_device(b, 31, False, torch.zeros(n, dtype=torch.int32), None, None)
    assert rt.count("purity_mask_kernel") == (n >= 65536)
    assert rt.count("launch ") == (3 if n >= 65536 else 2)
