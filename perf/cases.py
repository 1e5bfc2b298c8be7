"""Measured cases: the work that users of this engine have it do.

listed()            the cases; draw(rng) another one of the same ranges
prepare(case, seed) the inputs, on the GPU (host memory for the host-buffer call), and the
                    handle, batch, kept tiles or model that a program keeps
run(state)          one pass through the public entry points of hsmu_gb; returns C whole
exact(case, seed)   the same product's values in plain torch, 64 bits
work(case)          bytes and operations that one pass cannot do without

A case is {"kind": ..., sizes}.  Sparsity comes from the case (random graphs: its "graph" number), values
from the seed.  Kinds:

plain    C = A*A on the device (Engine.spgemm), for three families of matrices: "grid2d" (5-point
         Laplacian), "fem" (27-point stencil with dof x dof node blocks), "rmat" (power-law graph)
         and "random" (uniform columns, Poisson row lengths)
aat      C = A*A^T: the transpose on the device, then the product
tiled    C = A*B with B's bit tiles kept between products (arithmetic: fused multiply-add)
host     C = A*A from page-locked host arrays into page-locked host arrays
wide64   C = A*A with int64 row pointers, in row panels when a cap is given
learned  C = A*A through the learned row scheduler with the shipped model
galerkin a batch of AMG triple products P^T (A P), one graph launch for all
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "hsmu-spgemm_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import hsmu_gb  # noqa: E402
from hsmu_gb import learned  # noqa: E402

MAX_PRODUCTS = 2.5e9  # the largest listed case (R-MAT of 262,144 vertices) has about 2.9e9


def listed():
    return [
        # the smallest call: a coarse grid's operator squared; launches and host work only
        {"name": "lap2d_64", "kind": "plain", "family": "grid2d", "side": 64},
        # the benchmark's 5-point Laplacian
        {"name": "lap2d_256", "kind": "plain", "family": "grid2d", "side": 256},
        # the benchmark's finite-element product: 192,000 rows of 81 entries
        {"name": "fem_40_dof3", "kind": "plain", "family": "fem", "side": 40, "dof": 3},
        # an ordinary power-law graph squared
        {"name": "rmat_65536", "kind": "plain", "family": "rmat", "n": 65536, "ef": 16, "graph": 2},
        # the benchmark's headline product: R-MAT scale 18, edge factor 16
        {"name": "rmat_262144", "kind": "plain", "family": "rmat", "n": 262144, "ef": 16, "graph": 2},
        # unstructured sparsity: short rows whose products scatter over all columns
        {"name": "random_150001", "kind": "plain", "family": "random", "n": 150001, "lam": 12, "graph": 7},
        # the A*A^T mode (similarity, normal equations) on an odd-sized graph
        {"name": "aat_30011", "kind": "aat", "n": 30011, "ef": 16, "graph": 3},
        # repeated products against one operator: scalar 27-point rows, B converted once
        {"name": "tiled_fma_33", "kind": "tiled", "side": 33, "dof": 1},
        # a caller whose matrices live in host memory
        {"name": "host_fem_16_dof3", "kind": "host", "side": 16, "dof": 3},
        # 64-bit row pointers, several row panels
        {"name": "wide64_49999", "kind": "wide64", "n": 49999, "ef": 12, "graph": 5, "panel": 20000000},
        # the learned scheduler where it applies (warp-sized wide rows)
        {"name": "learned_32768", "kind": "learned", "n": 32768, "ef": 16, "graph": 2},
        # AMG set-up: one batch of Galerkin products of unequal grids
        {"name": "galerkin_20", "kind": "galerkin", "count": 20, "lo": 16, "hi": 96, "mix": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rmat_size(rng, lo, hi, ef_lo=4, ef_hi=24):
    """vertices and edge factor of a power-law graph whose square stays below the largest listed case
    (products of the squares of scales 15..18 at edge factor 16: about 44 n ef^2 (n / 262144)^0.45)"""
    while True:
        n, ef = _log(rng, lo, hi), rng.randint(ef_lo, ef_hi)
        if 44.0 * n * ef ** 2 * (n / 262144.0) ** 0.45 < MAX_PRODUCTS:
            return n, ef


def draw(rng):
    graph = rng.randint(0, 1 << 20)
    kind = rng.choice(["grid2d", "fem", "rmat", "random", "aat", "tiled", "host", "wide64", "learned", "galerkin"])
    if kind == "grid2d":
        return {"kind": "plain", "family": kind, "side": _log(rng, 24, 1024)}
    if kind == "fem":
        dof = rng.randint(1, 3)
        return {"kind": "plain", "family": kind, "side": _log(rng, 5, 40), "dof": dof}
    if kind == "rmat":
        n, ef = _rmat_size(rng, 1000, 200000)
        return {"kind": "plain", "family": kind, "n": n, "ef": ef, "graph": graph}
    if kind == "random":
        while True:
            n, lam = _log(rng, 2000, 1000000), _log(rng, 2, 40)
            if n * lam * lam < 1.2e8:
                return {"kind": "plain", "family": kind, "n": n, "lam": lam, "graph": graph}
    if kind == "aat":
        n, ef = _rmat_size(rng, 1000, 65536)
        return {"kind": kind, "n": n, "ef": ef, "graph": graph}
    if kind == "tiled":
        return {"kind": kind, "side": _log(rng, 6, 48), "dof": rng.randint(1, 2)}
    if kind == "host":
        return {"kind": kind, "side": _log(rng, 5, 20), "dof": rng.randint(1, 3)}
    if kind == "wide64":
        n, ef = _rmat_size(rng, 2000, 65536)
        return {"kind": kind, "n": n, "ef": ef, "graph": graph, "panel": rng.choice([0, 5000000, 20000000, 100000000])}
    if kind == "learned":
        n, ef = _rmat_size(rng, 8000, 65536, 8, 24)
        return {"kind": kind, "n": n, "ef": ef, "graph": graph}
    lo = rng.randint(6, 30)
    return {"kind": kind, "count": rng.randint(3, 20), "lo": lo, "hi": rng.randint(lo + 10, 96),
            "mix": graph}


# ------------------------------------------------------------------ matrices
class Mat:
    """CSR on the GPU: int32 row_ptr and col, float64 val, columns ascending in every row"""

    def __init__(self, M, N, rp, col, val):
        self.M, self.N, self.rp, self.col, self.val = M, N, rp, col, val


def _gen(seed, *more):
    """a generator on the GPU for this seed and purpose"""
    s = int(seed)
    for m in more:
        s = (s * 1000003 + int(m)) % (1 << 62)
    return torch.Generator(device="cuda").manual_seed(s)


def _from_keys(M, N, key, val=None):
    """sorted unique keys row * N + col -> Mat"""
    row = torch.div(key, N, rounding_mode="floor")
    rp = torch.zeros(M + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=M), 0, out=rp[1:])
    return Mat(M, N, rp.to(torch.int32), (key - row * N).to(torch.int32).contiguous(), val)


def _uniform(n, g, lo=-1.0, hi=1.0):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * (hi - lo) + lo


def _stencil(side, dims, dof, points27, g):
    """5-point (2-D) or 27-point (3-D) stencil with full dof x dof blocks, values uniform(-1, 1)"""
    nodes = side ** dims
    nid = torch.arange(nodes, device="cuda")
    coord = [nid // side ** d % side for d in range(dims)]
    steps = [(0,) * dims]
    if points27:
        steps = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    else:
        for d in range(dims):
            for s in (-1, 1):
                steps.append(tuple(s if e == d else 0 for e in range(dims)))
        steps.sort(key=lambda v: sum(v[d] * 2 ** (8 * d) for d in range(dims)))
    rows, cols = [], []
    for v in steps:
        ok = torch.ones(nodes, dtype=torch.bool, device="cuda")
        nb = nid.clone()
        for d in range(dims):
            c = coord[d] + v[d]
            ok &= (c >= 0) & (c < side)
            nb += v[d] * side ** d
        rows.append(nid[ok])
        cols.append(nb[ok])
    key = torch.sort(torch.cat(rows) * nodes + torch.cat(cols)).values
    r, c = torch.div(key, nodes, rounding_mode="floor"), key % nodes
    if dof > 1:
        e = torch.arange(dof, device="cuda")
        n = nodes * dof
        key = ((r[:, None, None] * dof + e[None, :, None]) * n + c[:, None, None] * dof + e[None, None, :]).reshape(-1)
        key = torch.sort(key).values
    m = _from_keys(nodes * dof, nodes * dof, key)
    m.val = _uniform(key.numel(), g)
    return m


def _rmat(n, ef, graph, g):
    """R-MAT graph on n vertices (a power of two, or one cropped to n), quadrant probabilities
    0.57/0.19/0.19/0.05, repeated edges merged, values uniform(0, 1)"""
    scale = max(1, (n - 1).bit_length())
    ne, gg = n * ef, _gen(graph, 11)
    row = torch.zeros(ne, dtype=torch.int64, device="cuda")
    col = torch.zeros(ne, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(ne, device="cuda", generator=gg)
        row = row * 2 + (r >= 0.76)
        col = col * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = (row < n) & (col < n)
    key = torch.unique(row[keep] * n + col[keep])
    m = _from_keys(n, n, key)
    m.val = _uniform(key.numel(), g, 0.0, 1.0)
    return m


def _random(n, lam, graph, g):
    """rows of Poisson(lam) uniform columns, values uniform(-1, 1)"""
    gg = _gen(graph, 13)
    k = torch.poisson(torch.full((n,), float(lam), device="cuda"), generator=gg).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
    col = torch.randint(0, n, (row.numel(),), device="cuda", generator=gg)
    key = torch.unique(row * n + col)
    m = _from_keys(n, n, key)
    m.val = _uniform(key.numel(), g)
    return m


def _poisson7(side, g):
    """7-point operator of a variable-coefficient problem on a side^3 grid"""
    return _stencil(side, 3, 1, False, g)


def _prolongator(side):
    """piecewise-constant 2x2x2 aggregation of a side^3 grid, and its transpose"""
    n, cs = side ** 3, (side + 1) // 2
    nid = torch.arange(n, device="cuda")
    agg = nid % side // 2 + cs * (nid // side % side // 2 + cs * (nid // (side * side) // 2))
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    P = _from_keys(n, cs ** 3, nid * cs ** 3 + agg, one)
    Pt = _from_keys(cs ** 3, n, torch.sort(agg * n + nid).values, one)
    return P, Pt


def _sides(case):
    r = np.random.default_rng(case["mix"])
    return [int(s) for s in r.integers(case["lo"], case["hi"] + 1, size=case["count"])]


def _matrix(case, seed):
    """the left operand of every kind but the batch"""
    kind = case.get("family", case["kind"])
    g = _gen(seed, 17)
    if kind == "grid2d":
        return _stencil(case["side"], 2, 1, False, g)
    if kind in ("fem", "tiled", "host"):
        return _stencil(case["side"], 3, case["dof"], True, g)
    if kind == "random":
        return _random(case["n"], case["lam"], case["graph"], g)
    return _rmat(case["n"], case["ef"], case["graph"], g)


# ------------------------------------------------------------------ passes
@functools.lru_cache(maxsize=None)
def _engine():
    """one handle for the program, as the library asks for (one per host thread)"""
    return hsmu_gb.Engine()


def _dev(m):
    return hsmu_gb.DeviceCSR.from_tensors(m.M, m.N, m.rp, m.col, m.val)


class _Array:
    """a library-owned device array, readable by torch without a copy; keeps its owner alive"""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _array(owner, ptr, n, typestr, dtype):
    if n == 0:
        return torch.empty(0, dtype=dtype, device="cuda")
    return torch.as_tensor(_Array(owner, ptr, n, typestr), device="cuda")


def _views(C, rp64=False):
    d = C.desc
    rp = _array(C, d.row_ptr, d.M + 1, "<i8" if rp64 else "<i4", torch.int64 if rp64 else torch.int32)
    return rp, _array(C, d.col, d.nnz, "<i4", torch.int32), _array(C, d.val, d.nnz, "<f8", torch.float64)


class _HostCSR:
    def __init__(self, m):
        self.M, self.N = m.M, m.N
        self.row_ptr, self.col, self.val = (x.cpu().pin_memory() for x in (m.rp, m.col, m.val))


def prepare(case, seed):
    eng = _engine()
    kind = case["kind"]
    s = {"kind": kind, "eng": eng}
    if kind == "galerkin":
        A, P, Pt = [], [], []
        for k, side in enumerate(_sides(case)):
            A.append(_dev(_poisson7(side, _gen(seed, 29, k))))
            p, pt = _prolongator(side)
            P.append(_dev(p))
            Pt.append(_dev(pt))
        s["batch"] = hsmu_gb.Batch(eng, hsmu_gb.BATCH_GALERKIN, A, P, Pt)
        return s
    m = _matrix(case, seed)
    if kind == "host":
        d = _dev(m)
        nnz = int(eng.row_nnz(d, d).sum())  # the program's output arrays, sized once
        s["A"] = _HostCSR(m)
        s["out"] = tuple(torch.empty(n, dtype=t, pin_memory=True)
                         for n, t in ((m.M + 1, torch.int32), (nnz, torch.int32), (nnz, torch.float64)))
        return s
    s["A"] = _dev(m)
    if kind == "tiled":
        b = _matrix(case, seed + 7919)
        s["B"] = _dev(b)
        s["tiles"] = hsmu_gb.BTiles(eng, s["B"])
    elif kind == "wide64":
        s["panel"] = case["panel"]
    elif kind == "learned":
        params, s["margin"], _ = learned.load()
        s["params"] = torch.from_numpy(params).cuda()
    return s


def run(s):
    eng, kind = s["eng"], s["kind"]
    if kind == "plain":
        return _views(eng.spgemm(s["A"], s["A"]))
    if kind == "aat":
        At = eng.transpose(s["A"])
        C = eng.spgemm(s["A"], At)
        return _views(C), _views(At)
    if kind == "tiled":
        return _views(eng.spgemm(s["A"], s["B"], tiles=s["tiles"], arith=hsmu_gb.ARITH_FMA))
    if kind == "host":
        return eng.spgemm_host(s["A"], s["A"], out=s["out"])
    if kind == "wide64":
        return _views(eng.spgemm64(s["A"], s["A"], max_panel_nnz=s["panel"]), rp64=True)
    if kind == "learned":
        return _views(eng.spgemm_learned(s["A"], s["A"], s["params"], s["margin"]))
    b = s["batch"]
    b.graph_launch()
    b.status()
    return [_views(b.result(p)) for p in range(b.n)]


# ------------------------------------------------------------------ 64-bit reference and work
def _products_per_row(A, B):
    blen = (B.rp[1:] - B.rp[:-1]).to(torch.int64)
    c = torch.zeros(A.col.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(blen[A.col.long()], 0, out=c[1:])
    return c[A.rp[1:].long()] - c[A.rp[:-1].long()]


def _blocks(rowprod, most):
    """consecutive rows with at most `most` products together (one row at least)"""
    cum = np.concatenate(([0], np.cumsum(rowprod.cpu().numpy())))
    lo = 0
    while lo < len(cum) - 1:
        hi = max(lo + 1, int(np.searchsorted(cum, cum[lo] + most, side="right")) - 1)
        yield lo, hi
        lo = hi


def _expand(A, B, lo, hi, values=True):
    """every intermediate product of rows lo..hi-1: keys (row - lo) * N + col, and values"""
    e0, e1 = int(A.rp[lo]), int(A.rp[hi])
    k = A.col[e0:e1].long()
    start = B.rp[k].long()
    length = B.rp[k + 1].long() - start
    row = torch.repeat_interleave(torch.arange(hi - lo, device="cuda"), (A.rp[lo + 1:hi + 1] - A.rp[lo:hi]).long())
    first = torch.cumsum(length, 0) - length
    src = torch.repeat_interleave(torch.arange(e1 - e0, device="cuda"), length)
    q = torch.arange(src.numel(), device="cuda") - first[src] + start[src]
    key = row[src] * B.N + B.col[q].long()
    return key, (A.val[e0:e1][src] * B.val[q] if values else None)


def _product(A, B):
    """A * B by expanding, sorting and summing the products, row block by row block"""
    rows, cols, vals = [], [], []
    for lo, hi in _blocks(_products_per_row(A, B), 6e7):
        key, v = _expand(A, B, lo, hi)
        key, order = torch.sort(key, stable=True)
        u, inv = torch.unique_consecutive(key, return_inverse=True)
        del key
        vals.append(torch.zeros(u.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, v[order]))
        cols.append((u % B.N).to(torch.int32))
        rows.append(torch.bincount(torch.div(u, B.N, rounding_mode="floor"), minlength=hi - lo))
    rp = torch.zeros(A.M + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.cat(rows), 0, out=rp[1:])
    return Mat(A.M, B.N, rp.to(torch.int32), torch.cat(cols), torch.cat(vals))


def _transpose(A):
    row = torch.repeat_interleave(torch.arange(A.M, device="cuda"), (A.rp[1:] - A.rp[:-1]).long())
    key, order = torch.sort(A.col.long() * A.M + row)
    return _from_keys(A.N, A.M, key, A.val[order])


def exact(case, seed):
    if case["kind"] == "galerkin":
        out = []
        for k, side in enumerate(_sides(case)):
            P, Pt = _prolongator(side)
            out.append((None, None, _product(Pt, _product(_poisson7(side, _gen(seed, 29, k)), P)).val))
        return out
    A = _matrix(case, seed)
    if case["kind"] == "aat":
        At = _transpose(A)
        return (None, None, _product(A, At).val), (None, None, At.val)
    if case["kind"] == "tiled":
        return None, None, _product(A, _matrix(case, seed + 7919)).val
    return None, None, _product(A, A).val


def _csr(M, nnz, ptr=4):
    return ptr * (M + 1) + 12 * nnz


def _size(A, B):
    """(products, nnz of A*B); the latter from every k-th row where there are many products"""
    rp = _products_per_row(A, B)
    total = int(rp.sum())
    step = max(1, int(total // 1.5e8))
    if step == 1:
        nnz = sum(int(torch.unique(_expand(A, B, lo, hi, False)[0]).numel()) for lo, hi in _blocks(rp, 6e7))
        return total, nnz
    pick = torch.arange(0, A.M, step, device="cuda")
    lens = (A.rp[1:] - A.rp[:-1]).long()[pick]
    srp = torch.zeros(pick.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=srp[1:])
    idx = torch.arange(int(srp[-1]), device="cuda") - torch.repeat_interleave(srp[:-1] - A.rp[:-1].long()[pick], lens)
    S = Mat(pick.numel(), A.N, srp.to(torch.int32), A.col[idx], None)
    srow = _products_per_row(S, B)
    seen = sum(int(torch.unique(_expand(S, B, lo, hi, False)[0]).numel()) for lo, hi in _blocks(srow, 6e7))
    return total, int(seen * (total / max(1, int(srow.sum()))))


def work(case):
    """A and B read once, C written once (CSR: 4 bytes per row pointer and column, 8 per value); a
    multiply and an add per intermediate product"""
    if case["kind"] == "galerkin":
        nbytes = flops = 0
        for side in _sides(case):
            A, (P, Pt) = _poisson7(side, _gen(0, 29, 0)), _prolongator(side)
            AP = _product(A, P)
            p2, nnz = _size(Pt, AP)
            # A*P is the pass's own: not counted
            nbytes += sum(_csr(m.M, m.col.numel()) for m in (A, P, Pt)) + _csr(Pt.M, nnz)
            flops += 2 * (int(_products_per_row(A, P).sum()) + p2)
        return {"bytes": nbytes, "flops": flops}
    A = _matrix(case, 0)
    B = _transpose(A) if case["kind"] == "aat" else A
    prods, nnz = _size(A, B)
    nbytes = _csr(A.M, A.col.numel()) + _csr(A.M, nnz, 8 if case["kind"] == "wide64" else 4)
    if case["kind"] == "aat":
        nbytes += _csr(B.M, B.col.numel())  # A^T is returned too
    if case["kind"] == "tiled":
        nbytes += _csr(A.M, A.col.numel())
    return {"bytes": nbytes, "flops": 2 * prods}
