"""Repeated entries found at load (csrc/gsofa_kernels.cu repeated_kernel): rows
out of order are told from rows that hold an id twice whatever their length, at
the edges of the warp's and the table's sizes; results against the oracle."""
import numpy as np
import pytest

from gsofatpds_b200 import gen
from tests.test_gpu_parity import check_full, ctx, oracle_full  # noqa: F401

pytestmark = pytest.mark.gpu

LENGTHS = (2, 31, 32, 33, 64, 1024, 1025, 4096, 4097, 9000)


def rows_of(order, twice=None):
    """A 10,000-row pattern with a core whose first rows have these lengths;
    order: sorts or shuffles a row; twice: (row, first, again) copies an entry."""
    n = 10000
    _, rp, col = gen.random_extra(n, 3, seed=41)
    rng, mix = np.random.default_rng(42), np.random.default_rng(43)
    beg, parts, at = np.zeros(n + 1, np.int64), [], 0
    for v in range(n):
        row = col[rp[v]:rp[v + 1]]
        if v < len(LENGTHS):
            row = np.union1d([v], rng.choice(n, LENGTHS[v], replace=False))[:LENGTHS[v]]
        row = order(mix, row)
        if twice and twice[0] == v:
            row = row.copy()
            row[twice[2]] = row[twice[1]]
        parts.append(row)
        at += row.size
        beg[v + 1] = at
    return beg[:-1].astype(np.int32), beg[1:].astype(np.int32), np.concatenate(parts).astype(np.int32)


def test_order_alone_changes_nothing(ctx):  # noqa: F811
    counts = []
    for order in (lambda mix, row: np.sort(row), lambda mix, row: mix.permutation(row)):
        t = rows_of(order)
        m = ctx.load_csr(*t)
        res = ctx.factor(m)
        check_full(res, *oracle_full(*t), l_rows=False)
        counts.append(res.counts)
        res.close()
        m.close()
    # both counted on top of what the hubs reach, which traverse_kernel does not do
    assert counts[0]["sources_chained"] == counts[1]["sources_chained"] > 10000


@pytest.mark.parametrize("row", range(len(LENGTHS)))
def test_one_entry_twice(ctx, row):  # noqa: F811
    n = LENGTHS[row]
    t = rows_of(lambda mix, r: mix.permutation(r), (row, 0, n - 1))
    m = ctx.load_csr(*t)
    res = ctx.factor(m)
    check_full(res, *oracle_full(*t), l_rows=False)
    res.close()
    m.close()
