"""A matrix most of whose sources reach no hub: its large searches would cost more
than traverse_kernel takes for all of it, and it is left to that kernel, alone, in a
captured batch and served; the same results, and not much slower."""
import numpy as np
import pytest

from gsofatpds_b200 import gen
from tests.test_gpu_parity import ctx  # noqa: F401

pytestmark = pytest.mark.gpu

TOTALS = ("fill_count", "nnz_l", "nnz_u", "edges_alg", "vertices_alg", "n_supernodes")


def same(a, b):
    for k in TOTALS:
        assert a.counts[k] == b.counts[k], k
    for f in ("row_counts", "digests"):
        for p, q in zip(getattr(a, f)().values(), getattr(b, f)().values()):
            np.testing.assert_array_equal(p, q)
    np.testing.assert_array_equal(a.lmask(), b.lmask())


def test_ordered_circuit(ctx):  # noqa: F811
    n, rp, col = gen.circuit_like()
    m = ctx.load_rowptr(rp, col)
    perm = ctx.order_hybrid(m)
    pm = ctx.permute(m, perm[0] if isinstance(perm, tuple) else perm)
    # traverse_kernel, by bottom-up sweeps that never set in
    walk = [ctx.factor(pm, bu_alpha=1, bu_min_source=n) for _ in range(2)]
    hubs = [ctx.factor(pm) for _ in range(2)]
    for r in hubs:
        same(r, walk[0])
    # the attempt is labels, the warps' searches and the first large ones: 0.05 to
    # 0.15 of the whole by the phases' times; without the rule it was 1.7
    took = [min(r.counts["ms_device"] for r in rs) for rs in (walk, hubs)]
    assert took[1] < 1.35 * took[0], took
    small = ctx.load_rowptr(*gen.random_extra(3000, 3, seed=3)[1:])
    alone = ctx.factor(small)
    b = ctx.batch([small, pm])
    for _ in range(2):
        b.run()
        same(b.result(0), alone)
        same(b.result(1), walk[0])
    b.close()
    for r in walk + hubs + [alone]:
        r.close()
    for x in (small, pm, m):
        x.close()
