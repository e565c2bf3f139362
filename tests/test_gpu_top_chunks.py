"""Meshes at the order from which the last separators' chunks have a launch of
their own, on a second stream: every count, digest and mask against
traverse_kernel's, which has no such launch, in a call and in a captured batch."""
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


@pytest.mark.parametrize("dims,stencil", [((255, 257), "5"), ((256, 256), "5"), ((300, 301), "9"), ((41, 40, 41), "7")])
def test_last_separators(ctx, dims, stencil):  # noqa: F811
    n, rp, col = gen.grid_nd(dims, stencil)
    m = ctx.load_rowptr(rp, col)
    small = ctx.load_rowptr(*gen.grid_nd((40, 40), "5")[1:])
    want = ctx.factor(m, chain=False)
    for kw in (dict(), dict(chunk_sources=1), dict(chunk_sources=3000), dict(global_bitmap=True)):
        got = ctx.factor(m, **kw)
        same(got, want)
        got.close()
    b = ctx.batch([small, m, m])
    for _ in range(2):
        b.run()
        same(b.result(1), want)
        same(b.result(2), want)
    b.close()
    want.close()
    for x in (small, m):
        x.close()
