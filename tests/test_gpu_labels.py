"""Hub labels (csrc/gsofa_hub.cu) against the oracle, bit for bit: the label
searches of one launch run in clusters of 1 to 16 CTAs, by how many matrices
share it, and labels of a random pattern are lowered many times."""
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
