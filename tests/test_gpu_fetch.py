"""The handoff's five arrays at block counts where they are small and lie close
together on the device: each against the oracle's patterns."""
import numpy as np
import pytest

from gsofatpds_b200 import gen
from oracle import oracle as O
from tests.test_gpu_parity import _supernodal_reference, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 63, 64, 65, 127, 128, 500, 1025])
@pytest.mark.parametrize("kind", ["diagonal", "random", "band"])
def test_small_handoff(ctx, n, kind):  # noqa: F811
    if kind == "diagonal":
        _, rp, col = gen.from_coo(n, np.arange(n), np.arange(n))
    elif kind == "random":
        _, rp, col = gen.random_extra(n, 2, seed=n)
    else:
        _, rp, col = gen.random_banded(n, bw=3, extra=0, seed=n)
    beg, end = gen.csr_to_beg_end(rp)
    r = O.rows(beg, end, col, pattern=True)
    _, flags = O.supernodes(r["nzU_ref"], r["lback"], 128)
    ref = _supernodal_reference(n, r, flags)
    m = ctx.load_rowptr(rp, col)
    res = ctx.factor(m, pattern=True)
    got = res.supernodal()
    for k, v in ref.items():
        np.testing.assert_array_equal(got[k], np.asarray(v), err_msg=k)
    res.close()
    m.close()
