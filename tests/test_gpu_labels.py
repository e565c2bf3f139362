"""Hub labels (csrc/gsofa_hub.cu) against the oracle, bit for bit: the label
searches of one launch run in clusters of 1 to 16 CTAs, by how many matrices
share it, and labels of a random pattern are lowered many times."""
import numpy as np
import pytest

from gsofatpds_b200 import gen
from tests.test_gpu_parity import check_full, ctx, oracle_full  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 4, 9, 20])
def test_every_cluster_width(ctx, count):  # noqa: F811
    ts = [gen.circuit_like(1500 + 37 * k, target_nnz=15000, seed=50 + k) for k in range(count)]
    mats = [ctx.load_rowptr(rp, col) for _, rp, col in ts]
    refs = []
    for n, rp, col in ts:
        beg, end = gen.csr_to_beg_end(rp)
        refs.append(oracle_full(beg, end, col))
    for _ in range(3):
        results = ctx.factor_batch(mats)
        for res, (r, rt) in zip(results, refs):
            check_full(res, r, rt, l_rows=False)
            res.close()
    for m in mats:
        m.close()


@pytest.mark.parametrize("name", ["circuit", "random", "banded", "dense"])
def test_labels_by_the_whole_gpu(ctx, name):  # noqa: F811
    """Labels in global memory, one launch a round: what orders above 900,000
    take, forced by the diagnostic option."""
    n, rp, col = {
        "circuit": lambda: gen.circuit_like(9000, target_nnz=80000, seed=8),
        "random": lambda: gen.random_extra(12000, 3, seed=61),
        "banded": lambda: gen.random_banded(4097, bw=5, extra=1, seed=6),
        "dense": lambda: gen.from_coo(1500, np.concatenate([np.arange(1500), np.full(1500, 900), np.arange(1500)]),
                                      np.concatenate([np.arange(1500), np.arange(1500), np.full(1500, 1100)])),
    }[name]()
    beg, end = gen.csr_to_beg_end(rp)
    r, rt = oracle_full(beg, end, col)
    m = ctx.load_rowptr(rp, col)
    chained = []
    for kw in (dict(), dict(global_bitmap=True), dict(global_bitmap=True, l_row_stats=True)):
        res = ctx.factor(m, **kw)
        check_full(res, r, rt, l_rows="l_row_stats" in kw)
        chained.append(res.counts["sources_chained"])
        res.close()
    assert len(set(chained)) == 1  # the same labels: none of them was left
    mats = [m, ctx.load_rowptr(*gen.random_extra(1500, 2, seed=62)[1:]), m]
    results = ctx.factor_batch(mats, global_bitmap=True)
    check_full(results[0], r, rt, l_rows=False)
    check_full(results[2], r, rt, l_rows=False)
    for res in results:
        res.close()
    for x in mats[:2]:
        x.close()


@pytest.mark.parametrize("seed", [8, 32])
def test_a_hub_that_is_given_up(ctx, seed):  # noqa: F811
    """Random patterns whose labels take more than 192 rounds for one of the
    first window's hubs: given up in the whole GPU's rounds (which end there),
    finished by the clusters (whose limit is higher once the set has settled)."""
    n, rp, col = gen.random_extra(20000, 3, seed=seed)
    beg, end = gen.csr_to_beg_end(rp)
    r, rt = oracle_full(beg, end, col)
    m = ctx.load_rowptr(rp, col)
    for kw in (dict(), dict(global_bitmap=True), dict(l_row_stats=True), dict(global_bitmap=True, l_row_stats=True)):
        res = ctx.factor(m, **kw)
        check_full(res, r, rt, l_rows="l_row_stats" in kw)
        res.close()
    m.close()
