"""Timed cases of the framework's public entry points.

A case is a dict of plain values.  ``listed()`` gives the fixed cases, ``draw``
one more of the same ranges, ``prepare`` what a program holds before the call
(a context, device-resident matrices, a prepared batch, a running server, host
arrays), ``run`` one pass through the public entry points and its results, and
``work`` the bytes a pass cannot do without.  Every output is a whole number:
structural counts, digests, flags, ids.

Matrices are the repository's own seeded generator families: 2D and 3D grids in
nested-dissection order (with one coupling in a hundred removed, which ones
depends on the seed, so that a mesh is not the same every time), random-banded
and random unsymmetric patterns, and the circuit-like pattern.
"""
import ctypes
import functools
import math

import numpy as np

from gsofatpds_b200 import _lib as C
from gsofatpds_b200 import gen
from gsofatpds_b200.api import Context

_COUNTS = ("fill_count", "nnz_l", "nnz_u", "nnz_lu", "n_supernodes", "edges_alg", "vertices_alg")
# ids a row in the supernodal form, at most: the size of a program's buffers
_HANDOFF_IDS = {"grid2d": 64, "grid3d": 160}


def listed():
    """The fixed cases, smallest work first within each entry point."""
    return [
        # a few hundred rows: a program that factors many tiny systems one by
        # one; launches and host work count
        dict(name="factor_banded_300", do="factor", family="banded", n=300, bw=5, extra=1),
        # a small planar mesh (a 45 x 45 five-point grid)
        dict(name="factor_grid2d_2k", do="factor", family="grid2d", n=2025, stencil=5),
        # an unsymmetric system of the size of the reference's bundled matrix,
        # with the optional per-row L counts
        dict(name="factor_banded_12k_lrows", do="factor", family="banded", n=11948, bw=9, extra=2,
             l_rows=True),
        # the random benchmark matrix: diagonal, tridiagonal, three columns a row
        dict(name="factor_random_20k", do="factor", family="random", n=20000, extra=3),
        # the 64^3 seven-point mesh of the benchmark
        dict(name="factor_grid3d_262k", do="factor", family="grid3d", n=262144, stencil=7),
        # the headline: the circuit-like matrix of the reference's test graph's shape
        dict(name="factor_circuit_659k", do="factor", family="circuit", n=659033),
        # a new matrix from host arrays through upload, factorization and
        # read-back: a 500 x 500 nine-point grid
        dict(name="load_factor_grid2d_250k", do="load_factor", family="grid2d", n=250000, stencil=9),
        # many matrices of uneven size in one prepared launch
        dict(name="batch_64", do="batch", count=64, nmin=2000, nmax=30000),
        # a burst of requests at a running server
        dict(name="serve_24", do="serve", count=24, nmin=1000, nmax=60000),
        # the structure a supernodal numeric factorization allocates from (40^3 mesh)
        dict(name="handoff_grid3d_64k", do="handoff", family="grid3d", n=64000, stencil=7),
        # fill-reducing ordering of a renumbered 64^3 mesh, and the reordered matrix
        dict(name="order_nd_grid3d_262k", do="order_nd", family="grid3d", n=262144, stencil=7),
        # the hybrid ordering, made for circuit-like patterns
        dict(name="order_hybrid_circuit_100k", do="order_hybrid", family="circuit", n=100000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _family(rng, name, lo, hi):
    """A matrix of the family, n spread over the logarithm of [lo, hi]."""
    c = dict(family=name, n=_log_int(rng, lo, hi))
    if name == "grid2d":
        c["stencil"] = rng.choice((5, 9))
    elif name == "grid3d":
        c["stencil"] = rng.choice((7, 27)) if c["n"] <= 60000 else 7
    elif name == "banded":
        c.update(bw=rng.randint(4, 32), extra=rng.randint(1, 4))
    elif name == "random":
        c["extra"] = rng.randint(2, 4)
    return c


def draw(rng):
    """One more case of the listed ranges (odd sizes among them)."""
    do = rng.choice(("factor",) * 6 + ("load_factor", "batch", "serve", "handoff", "order_nd",
                                       "order_hybrid"))
    if do == "batch":
        nmin = _log_int(rng, 500, 4000)
        return dict(do=do, count=rng.randint(8, 64), nmin=nmin,
                    nmax=_log_int(rng, 2 * nmin, 30000))
    if do == "serve":
        nmin = _log_int(rng, 500, 4000)
        return dict(do=do, count=rng.randint(4, 24), nmin=nmin,
                    nmax=_log_int(rng, 2 * nmin, 60000))
    if do == "handoff":
        return dict(do=do, **_family(rng, rng.choice(("grid2d", "grid3d")), 1000, 64000))
    if do == "order_nd":
        return dict(do=do, **_family(rng, rng.choice(("grid2d", "grid3d", "circuit")), 5000, 262144))
    if do == "order_hybrid":
        return dict(do=do, **_family(rng, rng.choice(("grid2d", "circuit")), 5000, 100000))
    if do == "load_factor":
        name = rng.choice(("grid2d", "grid3d", "banded", "random"))
        hi = {"grid2d": 250000, "grid3d": 150000, "banded": 20000, "random": 20000}[name]
        return dict(do=do, **_family(rng, name, 1000, hi))
    name = rng.choice(("grid2d", "grid3d", "banded", "random", "circuit"))
    lo, hi = {"grid2d": (300, 250000), "grid3d": (300, 262144), "banded": (300, 40000),
              "random": (300, 40000), "circuit": (20000, 659033)}[name]
    c = dict(do=do, **_family(rng, name, lo, hi))
    if c["n"] <= 20000 and rng.random() < 0.25:
        c["l_rows"] = True
    return c


# ---- inputs -----------------------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _grid(n, dims, stencil):
    side = max(2, int(round(n ** (1.0 / dims))))
    return gen.grid_nd((side,) * dims, str(stencil))


def _grid_with_gaps(n, dims, stencil, seed):
    """The grid less about 1 % of its couplings (i, j), (j, i)."""
    n, rowptr, col = _grid(n, dims, stencil)
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(rowptr))
    lo, hi = np.minimum(row, col), np.maximum(row, col)
    shift = 0x9E3779B97F4A7C15 * (seed % (1 << 31) + 1) % (1 << 64)
    h = (lo * n + hi).astype(np.uint64) + np.uint64(shift)
    h = (h ^ (h >> np.uint64(31))) * np.uint64(0xBF58476D1CE4E5B9)
    h ^= h >> np.uint64(29)
    keep = (row == col) | (h % np.uint64(100) != np.uint64(0))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(row[keep], minlength=n), out=ptr[1:])
    return n, ptr.astype(np.int32), np.ascontiguousarray(col[keep])


def _matrix(c, seed):
    """(n, rowptr, col) of the case's family."""
    f = c["family"]
    if f in ("grid2d", "grid3d"):
        return _grid_with_gaps(c["n"], 2 if f == "grid2d" else 3, c["stencil"], seed)
    if f == "banded":
        return gen.random_banded(c["n"], bw=c["bw"], extra=c["extra"], seed=seed)
    if f == "random":
        return gen.random_extra(c["n"], c["extra"], seed=seed)
    return gen.circuit_like(c["n"], target_nnz=int(c["n"] * 8.846), seed=seed)


def _mix(c, seed):
    """The batch's or the burst's matrices: sizes spread over the logarithm of
    [nmin, nmax] in no order, half 2D five-point grids, half random-banded."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(c["count"]):
        at = (0.6180339887498949 * (k + 1)) % 1.0  # the case alone says the sizes
        n = int(round(c["nmin"] * (c["nmax"] / c["nmin"]) ** at))
        s = int(rng.integers(1 << 30))
        if k % 2 == 0:
            out.append(_grid_with_gaps(n, 2, 5, s))
        else:
            out.append(gen.random_banded(n, bw=int(rng.integers(4, 17)), extra=int(rng.integers(1, 4)),
                                         seed=s))
    return out


@functools.lru_cache(maxsize=1)
def _context():
    return Context(0)  # one per program


class _Held:
    """What a program keeps between calls; its handles are closed with it."""

    def __init__(self, case):
        self.case = case
        self.ctx = _context()
        self.closing = []

    def __del__(self):
        for h in self.closing:
            h.close()


def prepare(case, seed):
    """The context and the handles or host arrays a program has in hand."""
    s = _Held(case)
    do = case["do"]
    if do in ("batch", "serve"):
        mats = _mix(case, seed)
        if do == "batch":
            s.mats = [s.ctx.load_rowptr(p, c) for _, p, c in mats]
            s.batch = s.ctx.batch(s.mats)
            s.closing = [s.batch] + s.mats
        else:
            s.requests = [(np.ascontiguousarray(p[:-1]), np.ascontiguousarray(p[1:]), c)
                          for _, p, c in mats]
            s.server = s.ctx.server(case["nmax"] + 1000, budget_bytes=6 << 30)
            s.closing = [s.server]
        return s
    n, rowptr, col = _matrix(case, seed)
    if do == "load_factor":
        s.host = (np.ascontiguousarray(rowptr[:-1]), np.ascontiguousarray(rowptr[1:]), col)
        return s
    s.mat = s.ctx.load_rowptr(rowptr, col)
    if do == "handoff":  # block starts, then pointers and ids of L and of U
        ids = int(n * _HANDOFF_IDS[case["family"]])
        s.bufs = [np.zeros(k, t) for k, t in ((n + 1, np.int32), (n + 1, np.int64), (ids, np.int32),
                                              (n + 1, np.int64), (ids, np.int32))]
    if do == "order_nd":  # an application's numbering: not the generator's order
        given = np.random.default_rng(seed).permutation(n).astype(np.int32)
        first, s.mat = s.mat, s.ctx.permute(s.mat, given)
        first.close()
    s.closing = [s.mat]
    return s


# ---- passes -----------------------------------------------------------------------


def _result(r, l_rows=False):
    """Everything a factorization gives but its timings."""
    out = {k: r.counts[k] for k in _COUNTS}
    out.update(r.row_counts(l_rows=l_rows))
    out.update(r.digests(l_rows=l_rows))
    out["supernode_flags"] = r.supernodes()[0]
    return out


def _results(rs):
    """The counts and per-row arrays of many results, one after another."""
    rows = [r.row_counts() for r in rs]
    out = {k: np.concatenate([x[k] for x in rows]) for k in rows[0]}
    out["counts"] = np.array([[r.counts[k] for k in _COUNTS] for r in rs], np.int64)
    out["supernode_flags"] = np.concatenate([r.supernodes()[0] for r in rs])
    return out


def _handoff(s):
    """The block form into the program's own buffers, as a numeric
    factorization takes it: the sizes first, then the arrays."""
    r = s.ctx.factor(s.mat, pattern=True)
    sizes = [ctypes.c_int64() for _ in range(3)]
    fn = C.load().gsofa_result_supernodal
    rc = fn(r._h, *[ctypes.byref(x) for x in sizes], None, None, None, None, None)
    nb, nl, nu = (x.value for x in sizes)
    if rc != C.OK or max(nl, nu) > s.bufs[2].shape[0]:
        raise RuntimeError("handoff: status %d, %d and %d ids" % (rc, nl, nu))
    rc = fn(r._h, None, None, None, *[b.ctypes.data_as(ctypes.c_void_p) for b in s.bufs])
    if rc != C.OK:
        raise RuntimeError("handoff: status %d" % rc)
    fill = r.counts["fill_count"]
    r.close()
    return [nb, nl, nu, fill] + s.bufs


def run(state):
    """One pass through the public entry points."""
    ctx, case = state.ctx, state.case
    do = case["do"]
    if do == "factor":
        l_rows = bool(case.get("l_rows"))
        r = ctx.factor(state.mat, l_row_stats=l_rows)
        out = _result(r, l_rows)
        r.close()
        return out
    if do == "load_factor":
        m = ctx.load_csr(*state.host)
        r = ctx.factor(m)
        out = _result(r)
        r.close()
        m.close()
        return out
    if do == "batch":
        state.batch.run()
        return _results([state.batch.result(i) for i in range(case["count"])])
    if do == "serve":
        tickets = [state.server.submit(*q) for q in state.requests]
        rs = [state.server.wait(t) for t in tickets]
        out = _results(rs)
        for r in rs:
            r.close()
        return out
    if do == "handoff":
        return _handoff(state)
    order = ctx.order_nd if do == "order_nd" else ctx.order_hybrid
    perm, stats = order(state.mat)
    ctx.permute(state.mat, perm).close()
    return [perm] + [stats[k] for k in ("rounds", "splits", "separator_vertices", "max_separator")]


def exact(case, seed):
    """No output is a rounded number: all are equal or wrong."""
    return None


# ---- what a pass cannot do without ---------------------------------------------------


def _entries(c):
    """Stored entries of the case's matrix, about."""
    f, n = c["family"], c["n"]
    per_row = {"grid2d": c.get("stencil", 5), "grid3d": c.get("stencil", 7),
               "banded": 1 + c.get("bw", 0) + c.get("extra", 0), "random": 3 + c.get("extra", 0),
               "circuit": 8.846}[f]
    return n * per_row


def work(case):
    """The matrix read once and the per-row results written once; the searches
    between them are integer work with no counted floating-point operations."""
    do = case["do"]
    if do in ("batch", "serve"):
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        n = case["count"] * (case["nmax"] - case["nmin"]) / (hi - lo)  # mean of a log-uniform size
        return {"bytes": n * (4 + 4 * 10) + n * 13, "flops": 0}
    n, nnz = case["n"], _entries(case)
    read = 4 * n + 4 * nnz
    if do in ("order_nd", "order_hybrid"):
        return {"bytes": 2 * read + 4 * n, "flops": 0}  # the permuted matrix is written too
    written = n * (29 + (12 if case.get("l_rows") else 0))
    return {"bytes": read + written, "flops": 0}
