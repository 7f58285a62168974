"""Performance cases of the library: the calls a program makes, over their real range of inputs.

A case names an operation and its input:

* ``multiply``: ``SpGEMM.multiply`` on device CSR matrices (C stays on the device),
* ``host``: the same call on host CSR matrices (copies in and out included),
* ``batch``: one ``Batch.run`` of a planned batch of independent products,
* ``sizes``: the per-row size estimates an application plans its memory with,
* ``train``: one optimiser step of the learned row-size estimator.

``listed()`` gives the named cases, ``draw(rng)`` more of the same ranges.
"""
import math

import torch

from research_b200 import estimator as E
from research_b200.matrices import laplacian_2d
from research_b200.ocean import MLP_FEATURES, MLP_PARAMS, Batch, DeviceCSR, SpGEMM, _check, _ptr, lib

DEV = "cuda"


def _case(name, op, family, n, deg, param=0, bits=32, learned=False, count=1):
    """family/n/deg/param: the input matrix (rows, entries per row, the family's
    width); bits: row-pointer width; learned: rows sized by the network;
    count: problems of a batch."""
    c = {"op": op, "family": family, "n": n, "deg": deg, "param": param, "bits": bits, "learned": learned,
         "count": count}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small banded system (one block of a multi-block solver): launches and read-backs count
        _case("band_small", "multiply", "banded", 1000, 8, 9),
        # 2D 5-point stencil squared: coarse-grid operators of multigrid
        _case("laplacian256", "multiply", "laplacian", 256, 5),
        # A * A^T of a short wide sparse matrix: normal equations, co-occurrence counts
        _case("rect_aat", "multiply", "rect", 262144, 12, 1048576),
        # unstructured uniform graph squared (two-hop neighbours): mid rows over wide column spans
        _case("uniform", "multiply", "uniform", 262144, 32),
        # wide band with an odd row count and the 64-bit row pointers torch programs hold
        _case("band_wide64", "multiply", "banded", 200003, 64, 256, bits=64),
        # dense diagonal blocks: high compaction, rows sized by the estimator instead of counted
        _case("block_learned", "multiply", "block", 131072, 64, 256, learned=True),
        # power-law graph squared, whole
        _case("rmat17", "multiply", "rmat", 131072, 16),
        # a 1/32 row sample of a 2^20-vertex power-law graph times the graph: one
        # row block of a product whose whole result is streamed block by block
        _case("rmat20_rows", "multiply", "rmat_rows", 1048576, 16, 32),
        # host buffers in, host buffers out
        _case("host_uniform", "host", "uniform", 50021, 16),
        # many independent problems of mixed families as one captured graph
        _case("batch16", "batch", "mixed", 65536, 0, learned=True, count=16),
        # row sizes of a power-law product too large to form
        _case("sizes_rmat21", "sizes", "rmat", 2097152, 24, learned=True),
        # one optimiser step of the row-size network
        _case("train_step", "train", "", 8192, 0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["multiply"] * 9 + ["host", "batch", "sizes", "train"])
    bits = 64 if rng.random() < 0.25 else 32
    if op == "train":
        return _case(None, op, "", _log(rng, 1000, 16384), 0)
    if op == "batch":
        return _case(None, op, "mixed", _log(rng, 8192, 65536), 0, learned=rng.random() < 0.5,
                     count=rng.randint(4, 16))
    if op == "sizes":
        return _case(None, op, rng.choice(["rmat", "uniform"]), _log(rng, 1 << 17, 1 << 21), rng.randint(8, 24),
                     bits=bits, learned=rng.random() < 0.5)
    if op == "host":
        return _case(None, op, rng.choice(["uniform", "banded"]), _log(rng, 1000, 60000), rng.randint(4, 16),
                     rng.randint(9, 65))
    family = rng.choice(["laplacian", "rect", "uniform", "banded", "block", "rmat", "rmat_rows"])
    learned = rng.random() < 0.3
    if family == "laplacian":
        return _case(None, op, family, rng.randint(40, 500), 5, bits=bits)
    if family == "rect":
        n = _log(rng, 4096, 262144)
        return _case(None, op, family, n, rng.randint(3, 14), n * rng.randint(2, 5) + rng.randint(0, 99), bits, learned)
    if family == "uniform":
        return _case(None, op, family, _log(rng, 1000, 262144), rng.randint(4, 32), 0, bits, learned)
    if family == "banded":
        return _case(None, op, family, _log(rng, 1000, 262144), rng.randint(4, 64), _log(rng, 3, 512), bits, learned)
    if family == "block":
        return _case(None, op, family, _log(rng, 1000, 262144), rng.randint(4, 64), _log(rng, 32, 1024), bits, learned)
    if family == "rmat":
        return _case(None, op, family, 1 << rng.randint(10, 17), rng.randint(4, 16), 0, bits, learned)
    return _case(None, op, family, 1 << rng.randint(18, 20), rng.randint(8, 16), rng.randint(32, 200), bits, learned)


# ---------------------------------------------------------------- inputs
# A case fixes the sparsity structure up to the order of A's rows, the seed
# draws that order and all values, so results of all seeds have the same size.

STRUCTURE = 7


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _csr(rows, cols, r, c, v):
    rp = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    return DeviceCSR(rows, cols, c.numel(), rp.to(torch.int32), c.to(torch.int32), v, 32)


def _coo(m):
    rp = m.rowptr.to(torch.int64)
    r = torch.repeat_interleave(torch.arange(m.rows, device=DEV), rp[1:] - rp[:-1])
    return r, m.col.to(torch.int64), m.val


def _roll(m, by):
    """m with its rows moved up cyclically by `by`: row order changes, neighbours stay neighbours."""
    by %= m.rows
    rp = m.rowptr.to(torch.int64)
    lens = torch.roll(rp[1:] - rp[:-1], -by)
    at = int(rp[by])
    out = torch.zeros_like(rp)
    out[1:] = torch.cumsum(lens, 0)
    return DeviceCSR(m.rows, m.cols, m.nnz, out.to(torch.int32), torch.roll(m.col, -at), torch.roll(m.val, -at), 32)


def _rect(rows, cols, lam):
    """(rows, columns) of a rows x cols matrix, Poisson(lam) entries per row at uniform columns."""
    g = _gen(STRUCTURE)
    k = torch.poisson(torch.full((rows,), float(lam), device=DEV), generator=g).to(torch.int64)
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), k)
    key = torch.unique(r * cols + torch.randint(0, cols, (r.numel(),), device=DEV, generator=g))
    return key // cols, key % cols


def _sample_rows(m, every):
    """rows / every random rows of m, in order."""
    pick = torch.randperm(m.rows, device=DEV, generator=_gen(STRUCTURE))[:max(1, m.rows // every)].sort().values
    to = torch.full((m.rows,), -1, dtype=torch.int64, device=DEV)
    to[pick] = torch.arange(pick.numel(), device=DEV)
    r, c, v = _coo(m)
    keep = to[r] >= 0
    return _csr(pick.numel(), m.cols, to[r[keep]], c[keep], v[keep])


def _widen(m):
    return DeviceCSR(m.rows, m.cols, m.nnz, m.rowptr.to(torch.int64), m.col, m.val, 64)


def _matrices(case, seed):
    """(A, B) of a product: a matrix with its rows in the seed's order, times the matrix (its transpose, for rect)."""
    f, n = case["family"], case["n"]
    g = _gen(seed)
    if f == "rect":
        r, c = _rect(n, case["param"], case["deg"])
        v = torch.randn(r.numel(), dtype=torch.float64, device=DEV, generator=g)
        at = torch.argsort(c * n + r)
        A, B = _csr(n, case["param"], r, c, v), _csr(case["param"], n, c[at], r[at], v[at])
    else:
        if f == "laplacian":
            B = DeviceCSR.from_host(laplacian_2d(n, n, STRUCTURE))
        else:
            B = E.generate("rmat" if f == "rmat_rows" else f, n, case["deg"], STRUCTURE, case["param"])
        B.val = torch.rand(B.nnz, dtype=torch.float64, device=DEV, generator=g) * 2.0 - 1.0
        A = _sample_rows(B, case["param"]) if f == "rmat_rows" else B
    A = _roll(A, seed * 7919 + 1)
    return (_widen(A), _widen(B)) if case["bits"] == 64 else (A, B)


def _batch_problems(case, seed):
    """(A, B) of mixed families in turn, rows log-uniform from 1000 to n, 4-32 entries per row."""
    specs = E.training_specs(case["count"], STRUCTURE, 1000, case["n"])
    return [_matrices(_case(None, "multiply", s.kind, s.n, s.deg, s.param), seed + i) for i, s in enumerate(specs)]


def _train_data(case, seed):
    """Normalised features and targets: log2 sizes between the rows' longest B row and their products."""
    g = _gen(seed)
    f = torch.randn((case["n"], MLP_FEATURES), device=DEV, generator=g)
    t = 8.0 + 2.0 * f[:, 1] + 0.5 * f[:, 2] * f[:, 5] + 0.1 * torch.randn(case["n"], device=DEV, generator=g)
    return f.contiguous(), t.contiguous()


def _config(case):
    return {"use_learned_estimator": True} if case["learned"] else None


def prepare(case, seed):
    op = case["op"]
    g = SpGEMM(_config(case))
    s = {"case": case, "g": g}
    if op == "batch":
        both = _batch_problems(case, seed)
        s["plan"] = Batch(g, [a for a, _ in both], [b for _, b in both])
    elif op == "train":
        s["x"], s["t"] = _train_data(case, seed)
        zero, one = [0.0] * MLP_FEATURES, [1.0] * MLP_FEATURES
        s["net"] = E.Network.initial(zero, one, seed=seed % (1 << 31))
        s["m1"], s["m2"], s["grad"] = (torch.zeros(MLP_PARAMS, device=DEV) for _ in range(3))
        s["loss"] = torch.zeros(1, device=DEV)
        s["step"] = 0
    else:
        if op == "sizes":
            A = E.generate(case["family"], case["n"], case["deg"], seed)
            s["A"] = s["B"] = _widen(A) if case["bits"] == 64 else A
        else:
            s["A"], s["B"] = _matrices(case, seed)
        if op == "host":
            s["A"], s["B"] = s["A"].download(), s["B"].download()
    return s


# ---------------------------------------------------------------- calls

class _Array:
    """A device array of a result, for torch (the result stays alive with it)."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr or 0), False), "shape": (n,), "typestr": kind, "version": 2}


def _tensors(c):
    o = c.view()

    def t(ptr, n, kind, dtype):
        return torch.as_tensor(_Array(c, ptr, n, kind), device=DEV) if n else torch.empty(0, dtype=dtype, device=DEV)
    rp = t(o.rowptr, o.rows + 1, "<i8" if o.rowptr_bits == 64 else "<i4", torch.int32)
    return [rp, t(o.col, o.nnz, "<i4", torch.int32), t(o.val, o.nnz, "<f8", torch.float64)]


def run(state):
    s, op = state, state["case"]["op"]
    if op == "multiply":
        return _tensors(s["g"].multiply(s["A"], s["B"]))
    if op == "host":
        c = s["g"].multiply(s["A"], s["B"])
        return [c.rowptr.view("int32"), c.col.view("int32"), c.val]
    if op == "batch":
        return [_tensors(c) for c in s["plan"].run()]
    if op == "sizes":
        return E.estimate(s["g"], s["A"], s["B"], "learned" if s["case"]["learned"] else "hll", True)
    net, n = s["net"], s["x"].shape[0]
    s["step"] += 1
    s["loss"].zero_()
    net.grad(s["g"], s["x"], s["t"], n, s["grad"], s["loss"])
    _check(lib().ocean_mlp_adam(s["g"]._h, _ptr(net.params), _ptr(s["m1"]), _ptr(s["m2"]), _ptr(s["grad"]), s["step"],
                                2e-3, 0.9, 0.999, 1e-8, None))
    return [net.params, s["m1"], s["m2"], s["loss"]]


# ---------------------------------------------------------------- work and tolerances

def _counts(case):
    """Expected (nnz(A), nnz(B), products, nnz(C)) of a product."""
    f, n, d, p = case["family"], case["n"], case["deg"], case["param"]
    if f == "laplacian":
        return 5 * n * n, 5 * n * n, 25 * n * n, 13 * n * n
    if f == "rect":
        z = n * d
        # two rows share a column: every entry meets the z / cols others of its column
        prod = z * (1.0 + z / p)
        return z, z, prod, prod - n * (d - 1)
    if f == "uniform":
        e = n * (1.0 - (1.0 - 1.0 / n) ** d)
        return n * e, n * e, n * e * e, n * n * (1.0 - math.exp(-e * e / n))
    if f in ("banded", "block"):
        w = 2 * p + 1 if f == "banded" else min(p, n)
        e = w * (1.0 - (1.0 - 1.0 / w) ** min(d, w))
        span = 4 * p + 1 if f == "banded" else w
        return n * e, n * e, n * e * e, n * span * (1.0 - math.exp(-e * e / span))
    # power law, fitted to the generator (2^17 and 2^20 rows, 16 entries per row)
    z = 0.93 * n * d
    prod = 2.09e10 * (n / 2.0 ** 20) ** 1.42 * (d / 16.0) ** 1.9
    out = min(9.7e9 * (n / 2.0 ** 20) ** 1.47 * (d / 16.0) ** 1.7, prod)
    if f == "rmat_rows":
        return z / p, z, prod / p, out / p
    return z, z, prod, out


def work(case):
    op = case["op"]
    if op == "train":
        n, h, x = case["n"], 64, MLP_FEATURES
        macs = (x * h + h * h + h) + (h + h * h) + (x * h + h * h + h)  # forward, dH, dW
        return {"bytes": n * 4 * (x + 1) + 8 * 4 * MLP_PARAMS, "flops": 2 * n * macs}
    if op == "batch":
        b = fl = 0.0
        for i in range(case["count"]):  # the families in turn, at the mean size and degree
            kind = E.FAMILIES[i % 4]
            n = (case["n"] - 1000) / math.log(case["n"] / 1000)
            w = work(_case(None, "multiply", kind, n, 18, 34 if kind == "banded" else 144))
            b, fl = b + w["bytes"], fl + w["flops"]
        return {"bytes": b, "flops": fl}
    za, zb, prod, out = _counts(case)
    n = case["n"]
    if op == "sizes":  # A * A by its structure alone
        return {"bytes": 4 * (za + n) + 4 * n, "flops": 2.0 * n * (16 * 64 + 64 * 64 + 64)}
    rp, cols = case["bits"] // 8, case["param"] if case["family"] == "rect" else n
    rows = n * n if case["family"] == "laplacian" else n // case["param"] if case["family"] == "rmat_rows" else n
    cols = rows if case["family"] == "laplacian" else cols
    return {"bytes": 12 * (za + zb) + rp * (rows + cols) + 12 * out + 4 * rows, "flops": 2 * prod}


def tolerance(case):
    if case["op"] == "train":
        # bf16 operands in the forward and backward products, sums in 32 bits
        return {"rel": 1e-2, "max": 0.05}
    if case["op"] == "sizes":
        # whole numbers from a bf16 network: a rounding may move a size by one
        return {"rel": 0.0, "differ": 0.01}
    # 64-bit sums in any order; the structure is the same entry by entry
    return {"rel": 1e-15, "max": 2e-13, "differ": 0.0}


# ---------------------------------------------------------------- plain torch

def _exact_product(A, B):
    """C = A * B by expanding, sorting and summing the products of row chunks."""
    arp, brp = A.rowptr.to(torch.int64), B.rowptr.to(torch.int64)
    acol, bcol = A.col.to(torch.int64), B.col.to(torch.int64)
    blen = brp[1:] - brp[:-1]
    per = torch.zeros(A.nnz + 1, dtype=torch.int64, device=DEV)
    per[1:] = torch.cumsum(blen[acol], 0)
    ends = per[arp]  # products before each row
    total = int(ends[-1])
    arow = torch.repeat_interleave(torch.arange(A.rows, device=DEV), arp[1:] - arp[:-1])
    counts = torch.zeros(A.rows, dtype=torch.int64, device=DEV)
    cols, vals, r0 = [], [], 0
    while r0 < A.rows:
        limit = int(ends[r0]) + (1 << 26)
        r1 = max(r0 + 1, min(A.rows, int(torch.searchsorted(ends, limit, right=True)) - 1))
        a0, a1 = int(arp[r0]), int(arp[r1])
        ent = torch.repeat_interleave(torch.arange(a0, a1, device=DEV), blen[acol[a0:a1]])
        p = torch.arange(ent.numel(), device=DEV) + int(ends[r0]) - per[ent] + brp[acol[ent]]
        key = (arow[ent] - r0) * B.cols + bcol[p]
        val = A.val[ent] * B.val[p]
        del ent, p
        key, inv = torch.unique(key, return_inverse=True)
        out = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, val)
        del inv, val
        counts[r0:r1] = torch.bincount(key // B.cols, minlength=r1 - r0)
        cols.append((key % B.cols).to(torch.int32))
        vals.append(out)
        r0 = r1
    rp = torch.zeros(A.rows + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(counts, 0)
    return [rp.to(torch.int32 if total < 2 ** 32 else torch.int64), torch.cat(cols), torch.cat(vals)]


def _exact_step(case, seed):
    """The first optimiser step in 64 bits."""
    x, t = (v.double() for v in _train_data(case, seed))
    zero, one = [0.0] * MLP_FEATURES, [1.0] * MLP_FEATURES
    p = E.Network.initial(zero, one, seed=seed % (1 << 31)).params.double().requires_grad_()
    h = E.H
    w1, w2, w3 = p[:E.OFF_B1].view(h, -1), p[E.OFF_W2:E.OFF_B2].view(h, h), p[E.OFF_W3:E.OFF_B3]
    y = torch.relu(x @ w1.T + p[E.OFF_B1:E.OFF_W2])
    y = torch.relu(y @ w2.T + p[E.OFF_B2:E.OFF_W3])
    err = y @ w3 + p[E.OFF_B3] - t
    loss = (err * err).sum()
    grad, = torch.autograd.grad(loss / case["n"], p)
    m1, m2 = 0.1 * grad, 0.001 * grad * grad
    new = p.detach() - 2e-3 * (m1 / 0.1) / (torch.sqrt(m2 / 0.001) + 1e-8)
    return [new, m1, m2, loss.detach().view(1)]


def exact(case, seed):
    if case["op"] == "sizes":
        return None
    if case["op"] == "train":
        return _exact_step(case, seed)
    if case["op"] == "batch":
        return [_exact_product(a, b) for a, b in _batch_problems(case, seed)]
    return _exact_product(*_matrices(case, seed))
