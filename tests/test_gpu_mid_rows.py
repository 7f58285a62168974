"""Forms of the mid-row kernels (dense, bucket, rank, hash by span; marked or
hashed symbolic rows): rows at the edges where one form gives way to the next,
against the oracle. Structure bit for bit, values within 1e-12 of
sum |a_ik * b_kj| (FP64 sums of at most 4096 terms in another order: below
4096 * 2^-53 = 4.6e-13 of it)."""
import numpy as np
import pytest

from oracle import oracle as O
from research_b200 import matrices as M
from research_b200.ocean import HostCSR

from test_gpu_parity import NUM_BINS, SYM_BINS, check, multiply_device

pytestmark = pytest.mark.gpu

CLASSES = {"hash_s": (128, 512), "hash_m": (256, 2048), "hash_l": (512, 4096)}  # threads, output entries


def _product(span, entries, length, repeat, seed, skew=False):
    """(A, B): B rows of `length` columns over exactly `span` columns, two in
    `repeat` of them shared by several rows; A rows take `entries` of B's rows, one
    fewer, and a third of them. skew: most columns are among the first 4096."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    pool = rng.choice(min(span, 4096) if skew else span, min(span, entries * length) if not skew else min(span, 4096),
                      replace=False)
    at = 0
    for i in range(entries):
        c = set()
        while len(c) < min(length, span):
            if repeat and len(c) < length // 2 and rng.random() < 2.0 / repeat:
                c.add(int(pool[rng.integers(0, min(64, pool.size))]))
            else:
                c.add(int(pool[at % pool.size]) if at < 2 * pool.size else int(rng.integers(0, span)))
                at += 1
        c = sorted(c)
        if i == 0:
            c[0], c[-1] = 0, span - 1
            c = sorted(set(c))
        rows += [i] * len(c)
        cols += c
    B = M.from_coo(entries, span + 3, rows, cols, rng.uniform(-1, 1, len(rows)))
    ar, ac = [], []
    for r, k in enumerate((entries, max(1, entries - 1), max(1, entries // 3))):
        ar += [r] * k
        ac += list(range(k))
    return M.from_coo(3, entries, ar, ac, rng.uniform(-1, 1, len(ar))), B


def _run(A, B, num, sym="bitmap", **cfg):
    C, _ = multiply_device(A, B, {"force_sym_bin": SYM_BINS[sym], "force_num_bin": NUM_BINS[num], **cfg})
    check(A, B, C)


@pytest.mark.parametrize("num", list(CLASSES))
@pytest.mark.parametrize("edge", [-1, 0, 1])
def test_products_at_the_register_limit(num, edge):
    # 4 products per thread: one B row less, exactly, one more
    threads, _ = CLASSES[num]
    for length, repeat in ((32, 8), (16, 3), (5, 4)):
        k = 4 * threads // length + edge
        A, B = _product(200000, k, length, repeat, 10 * k + length)
        if num == "hash_s" and np.unique(B.col).size > 512:
            A, B = _product(200000, min(k, 500 // length), length, repeat, 3)
        _run(A, B, num)


@pytest.mark.parametrize("span", [1, 2, 33, 1023, 1024, 1025, 4096, 4097, 8192, 8193, 65536, (1 << 20) - 1, 1 << 20,
                                  (1 << 20) + 1, 3 << 20])
@pytest.mark.parametrize("num", list(CLASSES))
def test_spans(num, span):
    _, cap = CLASSES[num]
    for entries, length in ((7, 60), (cap // 40, 37)):
        A, B = _product(span, entries, min(length, span), 5, span % 1000 + entries)
        _run(A, B, num)


@pytest.mark.parametrize("num", list(CLASSES))
def test_rows_that_fill_every_slot(num):
    # as many distinct columns as the class holds, every column once
    _, cap = CLASSES[num]
    rng = np.random.default_rng(cap)
    for span in (50000, 1 << 20):
        cols = np.sort(rng.choice(span, cap, replace=False))
        cols[0], cols[-1] = 0, span - 1
        order = np.argsort(rng.random(cap)) % 16
        B = M.from_coo(16, span, order, cols, rng.uniform(-1, 1, cap))
        A = M.from_coo(1, 16, np.zeros(16, int), np.arange(16), rng.uniform(-1, 1, 16))
        _run(A, B, num)


@pytest.mark.parametrize("num", list(CLASSES))
def test_skewed_columns_leave_the_bucket_form(num):
    # most products in a few buckets, and one column shared by every B row
    threads, _ = CLASSES[num]
    A, B = _product(1 << 19, 3 * threads // 32, 32, 2, 77, skew=True)
    _run(A, B, num)


@pytest.mark.parametrize("wf", [1, 2])
def test_forms_in_the_estimated_workflows(wf):
    # sizes estimated: rows that outgrow their slots go through the overflow list
    A = M.uniform_random(30000, 24, seed=4)
    C, st = multiply_device(A, A, {"force_workflow": wf, "estimate_scale": 0.4})
    check(A, A, C)
    assert st["decision"]["workflow"] == wf


@pytest.mark.parametrize("sym", list(CLASSES))
@pytest.mark.parametrize("words", [15, 16, 17])
def test_symbolic_marked_or_hashed(sym, words):
    # span words just below, at and above the products: marked or hashed
    A, B = _product(32 * 16 * words, 16, 16, 4, words)
    _run(A, B, "bitmap", sym)


def test_uneven_b_rows_take_the_balanced_enumeration():
    rng = np.random.default_rng(5)
    lens = np.r_[np.full(200, 2), 700, 300]
    r = np.repeat(np.arange(lens.size), lens)
    B = M.from_coo(lens.size, 90000, r, rng.integers(0, 90000, r.size), rng.uniform(-1, 1, r.size))
    A = M.from_coo(2, lens.size, np.repeat([0, 1], lens.size), np.tile(np.arange(lens.size), 2),
                   rng.uniform(-1, 1, 2 * lens.size))
    for num in ("hash_m", "hash_l"):
        for sym in CLASSES:
            _run(A, B, num, sym if sym != "hash_s" else "hash_m")


@pytest.mark.parametrize("num", list(CLASSES))
@pytest.mark.parametrize("edge", [-1, 0, 1])
def test_rows_of_many_short_entries(num, edge):
    # A rows at the 2 threads' worth of entries up to which lane groups walk them,
    # dense numeric and marked symbolic form
    threads, cap = CLASSES[num]
    A, B = _rows_of([2 * threads + edge] * 3, 2 * threads + 1, cap // 2, 4, edge + 5)
    _run(A, B, num, num)


def _narrow(rows, width, per_row, seed, repeat=False, length=40):
    """Product whose rows span exactly `width` columns: every A row references
    `per_row` B rows of `length` columns inside the width."""
    rng = np.random.default_rng(seed)
    nb = 64
    r, c = [], []
    for i in range(nb):
        k = np.sort(rng.choice(width, min(length, width), replace=False))
        if i == 0:
            k[0], k[-1] = 0, width - 1
        if repeat and i % 3 == 0:
            k[1::2] = k[0:len(k) - 1:2][:len(k[1::2])]  # every column twice
            k[0], k[-1] = 0, width - 1
            k = np.sort(k)
        r += [i] * len(k)
        c += list(k)
    B = M.from_coo(nb, width + 9, r, c, rng.uniform(-1, 1, len(r)), sum_duplicates=False)
    ar = np.repeat(np.arange(rows), per_row)
    ac = np.concatenate([np.r_[0, 1 + rng.choice(nb - 1, per_row - 1, replace=False)] for _ in range(rows)])
    return M.from_coo(rows, nb, ar, ac, rng.uniform(-1, 1, ar.size)), B


@pytest.mark.parametrize("width", [41, 1024, 1087, 1088, 1089, 4095, 4096, 4097])
@pytest.mark.parametrize("per_row,length", [(4, 33), (16, 8), (17, 8), (31, 40), (32, 40), (33, 40), (60, 7), (60, 9)])
def test_narrow_rows_run_a_warp_each(width, per_row, length):
    # spans at the limits of the numeric (1088) and symbolic (4096) narrow kernels,
    # A rows around one warp's entries, products around the 128 of the register
    # classes, B rows around the 8 entries that the narrow kernels ask for
    # (4096 equal rows: enough for a warp each)
    A, B = _narrow(4096, width, per_row, width + per_row, length=length)
    narrow = per_row * min(length, width) > 128 and length >= 8
    for a, b in ((A, B), (A.widened(), B.widened())):
        C, st = multiply_device(a, b)
        check(a, b, C)
        assert st["decision"]["numeric_narrow_rows"] == (A.rows if narrow and width <= 1088 else 0)
        assert st["decision"]["symbolic_narrow_rows"] == (A.rows if narrow and width <= 4096 else 0)


def _rows_of(counts, b_rows, width, length, seed):
    """A whose row r references counts[r] of the b_rows rows of B, each `length` columns of `width`."""
    rng = np.random.default_rng(seed)
    B = M.from_coo(b_rows, width, np.repeat(np.arange(b_rows), length), rng.integers(0, width, b_rows * length),
                   rng.uniform(-1, 1, b_rows * length))
    cols = np.concatenate([np.sort(rng.choice(b_rows, k, replace=False)) for k in counts])
    return M.from_coo(len(counts), b_rows, np.repeat(np.arange(len(counts)), counts), cols,
                      rng.uniform(-1, 1, cols.size)), B


@pytest.mark.parametrize("wf", [0, 1])
@pytest.mark.parametrize("rows,entries,light", [(3, 40000, 0), (300, 500, 0), (5, 20000, 6000), (0, 0, 6000)])
def test_heavy_or_few_narrow_rows_stay_in_blocks(wf, rows, entries, light):
    # rows with more products than a warp's share of the class, and classes with
    # too few rows for a warp each, run in their block class
    A, B = _rows_of([entries] * rows + [24] * light, 40000, 1000, 16, rows + 7)
    C, st = multiply_device(A, B, {"force_workflow": wf})
    check(A, B, C)
    assert st["decision"]["workflow"] == wf
    assert st["decision"]["numeric_narrow_rows"] == light
    assert st["decision"]["symbolic_narrow_rows"] == (light if wf == 0 else 0)


def test_small_skewed_product_has_no_narrow_rows():
    A = M.rmat(10, 8, seed=1)
    C, st = multiply_device(A, A)
    check(A, A, C)
    assert st["decision"]["numeric_narrow_rows"] == 0


@pytest.mark.parametrize("wf", [0, 1])
def test_narrow_rows_with_repeated_columns(wf):
    # B rows that hold a column twice: two lanes of one step meet
    A, B = _narrow(2200, 700, 40, 9, repeat=True)
    C, st = multiply_device(A, B, {"force_workflow": wf})
    check(A, B, C)
    assert st["decision"]["workflow"] == wf
    assert st["decision"]["numeric_narrow_rows"] == A.rows


@pytest.mark.parametrize("scale", [0.3, 1.0])
def test_narrow_rows_in_the_estimation_workflow(scale):
    A = M.block_diagonal(20000, 256, 64, seed=2)
    C, st = multiply_device(A, A, {"force_workflow": 1, "estimate_scale": scale})
    check(A, A, C)
    assert st["decision"]["workflow"] == 1


def test_narrow_rows_in_a_batch():
    # a captured plan runs its narrow rows a warp each, run after run
    from research_b200.ocean import Batch, DeviceCSR, SpGEMM
    ms = [M.banded(3000, 30, 16, seed=1), M.block_diagonal(2000, 100, 20, seed=2), M.uniform_random(1500, 14, seed=3)]
    for cfg in ({"force_workflow": 0}, {"use_learned_estimator": True}):
        g = SpGEMM(cfg)
        plan = Batch(g, [DeviceCSR.from_host(m) for m in ms])
        for _ in range(3):
            for m, c in zip(ms, plan.run()):
                check(m, m, c.download())
        plan.close()


@pytest.mark.parametrize("wf", [0, 1, 2])
@pytest.mark.parametrize("narrow_part", [0.0, 0.2, 0.3, 0.97, 1.0])
def test_rows_wider_than_a_bitmap_among_others(wf, narrow_part):
    # classes whose rows are all, mostly, partly or never wider than 2^20 columns:
    # the hash kernel takes the class whole from three quarters wide rows on
    rng = np.random.default_rng(int(100 * narrow_part) + wf)
    b_rows, cols, n = 6000, 3 << 20, 2000
    top = np.where(np.arange(b_rows) < b_rows // 2, 1 << 19, cols)  # the first half stays below 2^19 columns
    r = np.repeat(np.arange(b_rows), 16)
    B = M.from_coo(b_rows, cols, r, (rng.random(r.size) * top[r]).astype(np.int64), rng.uniform(-1, 1, r.size))
    k = rng.choice([12, 60, 200], n)  # one class each
    half = b_rows // 2
    ac = np.concatenate([np.sort(rng.choice(half, m, replace=False)) + (0 if i < narrow_part * n else half)
                         for i, m in enumerate(k)])
    A = M.from_coo(n, b_rows, np.repeat(np.arange(n), k), ac, rng.uniform(-1, 1, ac.size))
    for a, b in ((A, B), (A.widened(), B.widened())):
        C, st = multiply_device(a, b, {"force_workflow": wf})
        check(a, b, C)
        assert all(st["binning_2"][NUM_BINS[c]] for c in CLASSES)


def _special(A):
    """A with infinities, NaN and huge values among every 97th of its entries."""
    v = A.val.copy()
    at = np.arange(3, v.size, 97)
    v[at] = np.resize([np.inf, 1.0, np.nan, -np.inf, 1e300, 0.0, -1.0], at.size)
    return HostCSR(A.rows, A.cols, A.rowptr, A.col, v)


@pytest.mark.parametrize("form", ["narrow", "dense", "bucket", "rank", "wide", "items"])
def test_infinities_and_nan_stay_in_their_entries(form):
    # every accumulator is cleared whatever it holds, so the rows that a block or
    # a warp takes later are untouched
    if form == "narrow":
        A, cfg = M.banded(12000, 90, 20, seed=1), {}
    elif form == "items":
        A, cfg = M.rmat(14, 8, seed=2), {}
    else:
        cols = {"dense": 3000, "bucket": 60000, "rank": 60000, "wide": 3 << 20}[form]
        k = {"dense": 30, "bucket": 30, "rank": 60, "wide": 30}[form]
        A, B = _rows_of([k] * 4000, 3000, cols, 30, 3)
        cfg = {"force_sym_bin": SYM_BINS["bitmap"], "force_num_bin": NUM_BINS["hash_m"]}
    B = A if form in ("narrow", "items") else B
    A = _special(A)
    C, st = multiply_device(A, B, cfg)
    if form == "narrow":
        assert st["decision"]["numeric_narrow_rows"] > 11000
    if form == "items":
        assert st["decision"]["window_item_rows"] > 1000
    with np.errstate(all="ignore"):
        cp, cj, cx, ca = O.spgemm(A, B, with_abs=True)
        assert np.array_equal(C.rowptr.astype(np.uint64), cp) and np.array_equal(C.col, cj)
        nan, inf = np.isnan(cx), np.isinf(cx)
        assert nan.any() and inf.any()
        assert np.array_equal(np.isnan(C.val), nan) and np.array_equal(C.val[inf], cx[inf])
        fine = ~(nan | inf)
        assert (np.abs(C.val[fine] - cx[fine]) <= 1e-12 * ca[fine]).all()
