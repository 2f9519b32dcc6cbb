"""How a host SW batch, and its ranges that run at once, launch their work (on a runtime
that records, no GPU)."""
import numpy as np
import pytest

from fake_cuda import fake_path, rt  # noqa: F401
from genoaligner_gb300 import api, workloads

BLOCKS, WARPS = "sw16ck_kernelILi2ELb1E", "sw16ck_kernelILi2ELb0E"      # with, without whole-block items


def _call(n, length):
    """n pairs of one length, each side one buffer that every request shares."""
    a = workloads.random_bases(np.random.default_rng(1), length)
    off, lens = np.zeros(n, np.int64), np.full(n, length, np.int32)
    got = api.align_sw_batch_packed(a, off, lens, a, off, lens, scoring=(2, -3, 3, 1))
    assert got.status == api.Status.ok, got.error


def test_an_items_share_is_of_all_ranges(rt):
    _call(600, 1300)                                  # alone: few items, each on a block
    assert rt.count(BLOCKS) > 0 and rt.count(WARPS) == 0
    rt.clear()
    _call(20000, 1300)                                # 12 ranges: more items than the device has warps
    assert rt.count(WARPS) > 1 and rt.count(BLOCKS) == 0


def test_a_range_plans_in_small_blocks(rt):
    """Beside other ranges' persistent kernels a block of 1,024 threads finds no room."""
    _call(20000, 800)                                   # 6 ranges of 3,333 pairs
    assert rt.count("sp_scan_kernelILi256E") > 1
    assert rt.count("sp_small_kernel") == 0 and rt.count("sp_scan_kernelILi1024E") == 0
    rt.clear()
    _call(3333, 800)
    assert rt.count("sp_small_kernel") == 1 and rt.count("sp_scan_kernel") == 0
    rt.clear()
    _call(5000, 100)
    assert rt.count("sp_small_kernel") == 0 and rt.count("sp_scan_kernelILi1024E") == 1


def test_no_whole_block_phase_where_no_item_counts(rt):
    """Items above their share of a batch of more items than blocks, all narrow, stay on a
    warp each: the kernel without the whole-block phase runs them."""
    n = 2000
    rng = np.random.default_rng(2)
    a = workloads.random_bases(rng, 700)
    off, lens = np.zeros(n, np.int64), rng.integers(200, 700, n).astype(np.int32)
    for cigar in (True, False):
        rt.clear()
        got = api.align_sw_batch_packed(a, off, lens, a, off, lens, scoring=(2, -3, 3, 1), with_cigar=cigar)
        assert got.status == api.Status.ok, got.error
        with_phase, without = ((BLOCKS, WARPS) if cigar else ("sw16so_kernelILb1E", "sw16so_kernelILb0E"))
        assert rt.count(without) == 1 and rt.count(with_phase) == 0


@pytest.mark.parametrize("n,length,blocks", [(1600, 1300, True), (2200, 1300, False), (1600, 3000, True),
                                             (2000, 3000, True), (2300, 3000, False)])
def test_near_equal_items_of_a_full_device_stay_on_warps(rt, n, length, blocks):
    _call(n, length)                                    # n / 2 items, each above twice its share
    assert (rt.count(BLOCKS) > 0) == blocks and (rt.count(WARPS) > 0) == (not blocks)
