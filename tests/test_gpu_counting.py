"""The counting traversals (csrc/gsofa_chain.cu, csrc/gsofa_hub.cu) at the
sizes and patterns where their routes and tables change: alone searches up to
1,024 rows, hubs above, the chain for symmetric patterns, repeated entries and
matrices without a core; every count, digest, mask and supernode flag against
the oracle, bit for bit."""
import numpy as np
import pytest

from gsofatpds_b200 import gen
from tests.test_gpu_parity import check_full, ctx, oracle_full  # noqa: F401

pytestmark = pytest.mark.gpu


def renumbered(t, seed):
    n, rp, col = t
    p = np.random.default_rng(seed).permutation(n)
    rows = np.repeat(np.arange(n), np.diff(rp))
    return gen.from_coo(n, p[rows], p[col])


def blocks(*ts):
    """The matrices side by side on one diagonal."""
    r, c, off = [], [], 0
    for n, rp, col in ts:
        r.append(np.repeat(np.arange(n), np.diff(rp)) + off)
        c.append(col.astype(np.int64) + off)
        off += n
    return gen.from_coo(off, np.concatenate(r), np.concatenate(c))


def oriented(t):
    """A mesh with every coupling kept in one direction only, by its end ids'
    parity: unsymmetric, no strongly connected core."""
    n, rp, col = t
    rows = np.repeat(np.arange(n), np.diff(rp))
    keep = (rows == col) | ((rows + col) % 3 == 0) | (rows > col)
    return gen.from_coo(n, rows[keep], col[keep])


CASES = {
    # the alone search: one word, word edges, the largest order
    "one": lambda: gen.from_coo(1, [0], [0]),
    "alone_31": lambda: gen.random_extra(31, 2, seed=1),
    "alone_32": lambda: gen.random_extra(32, 2, seed=2),
    "alone_33": lambda: gen.random_extra(33, 2, seed=3),
    "alone_mesh_900": lambda: gen.grid_nd((30, 30), "9"),
    "alone_1024": lambda: gen.random_banded(1024, bw=3, extra=1, seed=4),
    # hubs: the smallest order, windows and words at their edges
    "hub_1025": lambda: gen.random_extra(1025, 3, seed=5),
    "hub_4095": lambda: gen.random_banded(4095, bw=5, extra=1, seed=6),
    "hub_4097": lambda: gen.circuit_like(4097, target_nnz=36000, seed=7),
    "hub_circuit_9000": lambda: gen.circuit_like(9000, target_nnz=80000, seed=8),
    # rows longer than one step of a warp (128 entries) and a dense row and column
    "hub_dense_row": lambda: gen.from_coo(
        3000, np.concatenate([np.arange(3000), np.full(3000, 1700), np.arange(3000)]),
        np.concatenate([np.arange(3000), np.arange(3000), np.full(3000, 2100)])),
    # no core: left to the chain
    "band_only": lambda: gen.random_banded(5000, bw=2, extra=0, seed=9),
    "oriented_mesh": lambda: oriented(gen.grid_nd((70, 70), "5")),
    # the chain: word edges, dense base, two interleaved cores, a renumbered mesh
    "mesh_1156": lambda: gen.grid_nd((34, 34), "5"),
    "mesh_17_cubed": lambda: gen.grid_nd((17, 17, 17), "27"),
    "two_meshes": lambda: renumbered(blocks(gen.grid_nd((40, 40), "9"), gen.grid_nd((41, 39), "5")), 10),
    "mesh_renumbered": lambda: renumbered(gen.grid_nd((45, 40), "5"), 11),
    "empty_rows": lambda: gen.from_coo(1500, np.arange(0, 1500, 3), np.arange(0, 1500, 3)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_counts_against_the_oracle(ctx, name):  # noqa: F811
    n, rp, col = CASES[name]()
    beg, end = gen.csr_to_beg_end(rp)
    m = ctx.load_rowptr(rp, col)
    r, rt = oracle_full(beg, end, col)
    # the default shape, one chunk per CTA and short ones, bitmaps in global memory
    for kw in (dict(), dict(chunk_sources=1000, threads_per_source=512), dict(chunk_sources=37),
               dict(global_bitmap=True), dict(l_row_stats=True)):
        res = ctx.factor(m, **kw)
        check_full(res, r, rt, l_rows="l_row_stats" in kw)
        res.close()
    m.close()


@pytest.mark.parametrize("n", [700, 2500])
def test_repeated_entries(ctx, n):  # noqa: F811
    """Rows out of order with entries twice: nz_row_U counts each."""
    rng = np.random.default_rng(n)
    _, rp, col = gen.random_extra(n, 3, seed=12)
    parts, beg, end, at = [], np.zeros(n, np.int32), np.zeros(n, np.int32), 0
    for v in range(n):
        row = rng.permutation(np.concatenate([col[rp[v]:rp[v + 1]]] * (2 if v % 5 == 0 else 1)))
        beg[v], end[v] = at, at + row.size
        parts.append(row)
        at += row.size
    col = np.concatenate(parts).astype(np.int32)
    m = ctx.load_csr(beg, end, col)
    r, rt = oracle_full(beg, end, col)
    res = ctx.factor(m, l_row_stats=True)
    check_full(res, r, rt)
    res.close()
    m.close()


def test_batch_of_every_route(ctx):  # noqa: F811
    """One captured launch over matrices of every route, run twice."""
    ts = [CASES[k]() for k in sorted(CASES)]
    mats = [ctx.load_rowptr(rp, col) for _, rp, col in ts]
    alone = [ctx.factor(m) for m in mats]
    b = ctx.batch(mats)
    for _ in range(2):
        b.run()
        for i, a in enumerate(alone):
            x = b.result(i)
            for k in ("fill_count", "nnz_l", "nnz_u", "edges_alg", "vertices_alg", "n_supernodes"):
                assert x.counts[k] == a.counts[k], (sorted(CASES)[i], k)
            for f in ("row_counts", "digests"):
                for p, q in zip(getattr(x, f)().values(), getattr(a, f)().values()):
                    np.testing.assert_array_equal(p, q)
            np.testing.assert_array_equal(x.lmask(), a.lmask())
    b.close()
    for a in alone:
        a.close()
    for m in mats:
        m.close()
