"""More matrices in one launch than a second grid dimension has indexes for
jobs (8 a matrix, 65,535): one unsymmetric matrix with a hub among 8,199 small
ones, plain and captured, against the oracle."""
import pytest

from gsofatpds_b200 import gen
from tests.test_gpu_parity import check_full, ctx, oracle_full  # noqa: F401

pytestmark = pytest.mark.gpu


def test_8200_matrices_in_one_launch(ctx):  # noqa: F811
    small = [gen.random_extra(5 + k, 1, seed=70 + k) for k in range(7)]
    ts = [small[k % 7] for k in range(8199)] + [gen.circuit_like(1100, target_nnz=11000, seed=3)]
    refs = []
    for n, rp, col in small + ts[-1:]:
        beg, end = gen.csr_to_beg_end(rp)
        refs.append(oracle_full(beg, end, col))
    mats = [ctx.load_rowptr(rp, col) for _, rp, col in ts]
    totals = [int(r["nnzU"].sum()) for r, _ in refs]
    which = [k % 7 for k in range(8199)] + [7]
    full = [0, 1, 2, 3, 4, 5, 6, 4099, 8198, 8199]
    for kw in (dict(), dict(l_row_stats=True)):
        results = ctx.factor_batch(mats, **kw)
        assert [res.counts["nnz_u"] for res in results] == [totals[w] for w in which]
        for i in full:
            check_full(results[i], *refs[which[i]], l_rows="l_row_stats" in kw)
        for res in results:
            res.close()
    b = ctx.batch(mats)
    b.run()
    assert [b.result(i).counts["nnz_u"] for i in range(len(mats))] == [totals[w] for w in which]
    for i in full:
        check_full(b.result(i), *refs[which[i]], l_rows=False)
    b.close()
    for m in mats:
        m.close()
