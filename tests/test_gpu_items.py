"""Window items of the numeric bitmap class (k_item_plan, k_num_items): rows
with saved bitmaps cut by entries (more than 10240) and by words (more than
2^19 columns), rows at the span where every row becomes items (2^18 columns),
heavy rows among wide light ones, more A entries than one chunk (1024) and than
the quarter search (256), 32- and 64-bit row pointers, row chunks of the
host-buffer pipeline. Structure must match the oracle bit for bit, values
within 1e-12 * sum |a*b| (at most 3000 FP64 terms per entry in another order:
below 3000 * 2^-53 = 3.4e-13 of it)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from research_b200 import matrices as M
from research_b200.ocean import DeviceCSR, SpGEMM

from test_gpu_parity import NUM_BINS, SYM_BINS, check, multiply_device
from test_gpu_windows import heavy_mix

pytestmark = pytest.mark.gpu

FORCE = {"force_sym_bin": SYM_BINS["bitmap"], "force_num_bin": NUM_BINS["bitmap"], "force_workflow": 0}


@pytest.mark.parametrize("cols", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, 1 << 20])
@pytest.mark.parametrize("wide_pointers", [False, True])
def test_power_law_rows(cols, wide_pointers):
    A, B = heavy_mix(b_rows=6000, cols=cols, seed=cols % 97)
    if wide_pointers:
        A, B = A.widened(), B.widened()
    C, st = multiply_device(A, B)
    check(A, B, C)
    assert st["decision"]["bitmap_cache_used_bytes"] > 0
    assert int(np.diff(C.rowptr.astype(np.int64)).max()) > 20480  # rows of several items
    d = st["decision"]
    assert 0 < d["window_item_rows"] < d["window_items"]
    if cols <= 1 << 18:  # every row with a saved bitmap
        assert d["window_item_rows"] == st["binning_1"][SYM_BINS["bitmap"]]


@pytest.mark.parametrize("span", [64, 2048, 2049, 1 << 18, (1 << 19) + 1, 1 << 20])
@pytest.mark.parametrize("entries", [1, 255, 256, 257, 1025])
def test_item_edges(span, entries):
    # rows of `entries` B rows of 9 columns and single-entry rows beside them, in
    # numbers that let their bitmaps be saved and items be launched: 1100 copies
    # of the row up to 2049 columns, one and a row of 12000 products beyond
    rng = np.random.default_rng(span + entries)
    r = np.repeat(np.arange(entries), 9)
    c = rng.integers(0, span, r.size)
    c[0], c[-1] = 0, span - 1
    whole, extra = (1100, 0) if span <= 2049 else (1, 20)
    for i in range(extra):
        r = np.r_[r, np.full(600, entries + i)]
        c = np.r_[c, rng.choice(span, 600, replace=False)]
    B = M.from_coo(entries + extra, span, r, c, rng.uniform(-1, 1, r.size))
    parts = [np.arange(entries)] * whole + [[0], [entries - 1]] + [entries + np.arange(extra)] * bool(extra)
    ar = np.repeat(np.arange(len(parts)), [len(k) for k in parts])
    A = M.from_coo(len(parts), entries + extra, ar, np.concatenate(parts), rng.uniform(-1, 1, ar.size))
    C, st = multiply_device(A, B, FORCE)
    check(A, B, C)
    prod, lo, hi = O.row_stats(A, B)
    prod, width = prod.astype(np.int64), hi.astype(np.int64) - lo.astype(np.int64) + 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cut = (width <= 1 << 18) | (prod > prod.sum() // (4 * sms))
    words = -(-width[cut] // 64)
    d = st["decision"]
    assert d["bitmap_cache_used_bytes"] > 0 and d["window_item_rows"] == cut.sum()
    # an item holds at most 256 groups of 32 words, and (here) no row more than 10240 entries
    most = O.symbolic(A, B).max()
    assert d["window_items"] == (-(-words // 8192)).sum() if most <= 10240 else d["window_items"] > cut.sum()


def test_items_hold_at_most_their_slots():
    # one dense row: every column of 2^18, so the cuts fall at the slot limit
    rng = np.random.default_rng(3)
    span = 1 << 18
    cols = rng.permutation(span)
    B = M.from_coo(64, span, np.arange(span) % 64, cols, rng.uniform(-1, 1, span))
    A = M.from_coo(2, 64, np.r_[np.zeros(64, int), np.ones(3, int)], np.r_[np.arange(64), 1, 5, 9],
                   rng.uniform(-1, 1, 67))
    C, _ = multiply_device(A, B)
    check(A, B, C)
    assert C.nnz > span


@pytest.mark.parametrize("scale,per_row,items", [(13, 8, False), (14, 8, True)])
def test_few_rows_of_one_item_run_whole(scale, per_row, items):
    # a few dozen rows of at most 8192 entries with a saved bitmap: no items; thousands: items
    A = M.rmat(scale, per_row, seed=2)
    C, st = multiply_device(A, A)
    check(A, A, C)
    assert st["decision"]["bitmap_cache_used_bytes"] > 0
    assert (st["decision"]["window_item_rows"] > 0) == items


@pytest.mark.parametrize("chunks", [2, 5])
def test_items_in_the_host_pipeline(chunks):
    A, B = heavy_mix(b_rows=6000, cols=1 << 18, seed=8)
    g = SpGEMM({"host_pipeline_chunks": chunks, "host_pipeline_min_products": 1, "small_problem_nnz": 0})
    C = g.multiply(A, B)
    check(A, B, C)
    d = g.get_stats()["decision"]
    assert d["host_pipeline_chunks"] == chunks and d["window_item_rows"] > 0


def test_growing_bitmaps_are_not_allocated_again_each_time():
    # the second product's bitmaps take 5% more than the first's
    rng = np.random.default_rng(4)
    b_rows, cols, n, k = 2000, 1 << 18, 2000, 60
    top = np.where(np.arange(b_rows) < b_rows // 2, 1 << 17, int(1.05 * (1 << 17)))
    r = np.repeat(np.arange(b_rows), 300)
    dB = DeviceCSR.from_host(M.from_coo(b_rows, cols, r, (rng.random(r.size) * top[r]).astype(np.int64),
                                        rng.uniform(-1, 1, r.size)))
    ac = np.concatenate([np.sort(rng.choice(b_rows // 2, k, replace=False)) for _ in range(n)])
    first, second = (DeviceCSR.from_host(M.from_coo(n, b_rows, np.repeat(np.arange(n), k), ac + shift,
                                                    rng.uniform(-1, 1, ac.size))) for shift in (0, b_rows // 2))
    warm, g = SpGEMM(), SpGEMM()
    warm.multiply(second, dB).free()  # the pool of C holds enough from here on
    words, free = [], []
    for A in (first, second):
        g.multiply(A, dB).free()
        torch.cuda.synchronize()
        words.append(g.get_stats()["decision"]["bitmap_cache_bytes"])
        free.append(torch.cuda.mem_get_info()[0])
    assert 1.02 * words[0] < words[1] < 1.1 * words[0]
    assert free[1] == free[0]
