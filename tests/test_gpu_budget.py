"""Memory budgets: a call that fits with traverse_kernel's workspace is never
refused because the counting traversals would like more of it, nor because an
earlier call's workspace is kept."""
import numpy as np
import pytest

from gsofatpds_b200 import Context, gen
from tests.test_gpu_parity import ctx  # noqa: F401

pytestmark = pytest.mark.gpu

MATRICES = {
    "random": lambda: gen.random_extra(20000, 3, seed=21),
    "circuit": lambda: gen.circuit_like(9000, target_nnz=80000, seed=22),
    "mesh": lambda: gen.grid_nd((100, 90), "9"),
}


def answer(res, l_rows, pattern):
    out = [res.counts[k] for k in ("fill_count", "nnz_l", "nnz_u", "n_supernodes")]
    arrays = list(res.row_counts(l_rows=l_rows).values()) + list(res.digests(l_rows=l_rows).values())
    if pattern:
        arrays += list(res.pattern_u()) + list(res.pattern_l())
    return out, [a for a in arrays if a is not None]


def same(a, b):
    assert a[0] == b[0] and len(a[1]) == len(b[1])
    for x, y in zip(a[1], b[1]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("name", sorted(MATRICES))
@pytest.mark.parametrize("kw", [dict(), dict(l_row_stats=True), dict(pattern=True)],
                         ids=["plain", "l_rows", "pattern"])
def test_tight_budget(ctx, name, kw):  # noqa: F811
    _, rp, col = MATRICES[name]()
    l_rows, pattern = "l_row_stats" in kw, "pattern" in kw
    m = ctx.load_rowptr(rp, col)
    ref = ctx.factor(m, **kw)
    want = answer(ref, l_rows, pattern)
    ref.close()
    m.close()
    # what traverse_kernel (without chained starts) keeps for eight CTAs
    with Context(0) as c:
        m = c.load_rowptr(rp, col)
        matrix = c.memory_used()
        res = c.factor(m, sources_in_flight=8, chain=False, **kw)
        used = c.memory_used()
        res.close()
        m.close()
    with Context(0, budget_bytes=used + (64 << 10)) as c:
        m = c.load_rowptr(rp, col)
        for _ in range(2):
            res = c.factor(m, sources_in_flight=8, **kw)
            same(answer(res, l_rows, pattern), want)
            res.close()
        m.close()
    # with room for a second matrix, which kept workspace gives way to
    with Context(0, budget_bytes=used + matrix + (64 << 10)) as c:
        m = c.load_rowptr(rp, col)
        res = c.factor(m, sources_in_flight=8, **kw)
        m2 = c.load_rowptr(rp, col)
        res.close()
        res = c.factor(m2, sources_in_flight=8, **kw)
        same(answer(res, l_rows, pattern), want)
        res.close()
        m2.close()
        m.close()


def test_tight_budget_batch(ctx):  # noqa: F811
    ts = [MATRICES[k]() for k in sorted(MATRICES)]
    mats = [ctx.load_rowptr(rp, col) for _, rp, col in ts]
    want = []
    for m in mats:
        res = ctx.factor(m)
        want.append(answer(res, False, False))
        res.close()
        m.close()
    with Context(0) as c:
        mats = [c.load_rowptr(rp, col) for _, rp, col in ts]
        b = c.batch(mats, sources_in_flight=8, chain=False)
        used = c.memory_used()
        b.close()
        for m in mats:
            m.close()
    with Context(0, budget_bytes=used + (64 << 10)) as c:
        mats = [c.load_rowptr(rp, col) for _, rp, col in ts]
        b = c.batch(mats, sources_in_flight=8)
        for _ in range(2):
            b.run()
            for i, w in enumerate(want):
                same(answer(b.result(i), False, False), w)
        b.close()
        for m in mats:
            m.close()
