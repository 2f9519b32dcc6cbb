"""Plain WFA batches on either side of the size at which a kernel sets the purity flags,
through the allocating and the non-allocating entry, with bytes other than A, C, G, T
at the sides' ends: equal to the oracle."""
import ctypes

import numpy as np
import pytest

import oracle
from genoaligner_gb300 import api, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 65536])
@pytest.mark.parametrize("smax", [31, 520])
def test_purity_of_every_pair(n, smax):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    lens = rng.integers(1, 70, n)
    ends = np.cumsum(lens)
    buf = workloads.random_bases(rng, int(ends[-1]))
    other = buf.copy()
    other[rng.random(other.size) < 0.03] = ord("C")
    other[ends[::7] - 1] = ord("N")                    # the last byte of every seventh text
    buf[ends[::11] - 1] = ord("n")
    off = (ends - lens).astype(np.int64)
    pats = [buf[o:e].tobytes() for o, e in zip(off, ends)]
    txts = [other[o:e].tobytes() for o, e in zip(off, ends)]
    want = oracle.wfa_batch(pats, txts, smax=smax, with_cigar=False, max_smax=4096).score
    lens = lens.astype(np.int32)
    b = api.DeviceBatchT(buf, off, lens, other, off, lens, device="cuda")
    sc = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    api.wfa_device(b, smax, False, sc, None, None)
    assert np.array_equal(sc.cpu().numpy(), want)
    f = api.load().ga_wfa_device_noalloc
    f.argtypes = [ctypes.POINTER(api.DeviceBatch), ctypes.c_int32, ctypes.c_int32] + 4 * [ctypes.c_void_p] + [
        ctypes.POINTER(ctypes.c_char_p)]
    f.restype = ctypes.c_int32
    sc.fill_(-7)
    torch.cuda.synchronize()
    err = ctypes.c_char_p()
    assert f(ctypes.byref(b.c), smax, 0, sc.data_ptr(), None, None, None, ctypes.byref(err)) == api.GA_OK, err.value
    torch.cuda.synchronize()
    assert np.array_equal(sc.cpu().numpy(), want)
