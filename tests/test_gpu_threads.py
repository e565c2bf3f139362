"""Contexts of their own in several threads: calls of very different sizes at
the same time, whose launches ask for different amounts of shared memory."""
import threading

import numpy as np
import pytest

from gsofatpds_b200 import Context, gen

pytestmark = pytest.mark.gpu

SIZES = [
    lambda: gen.random_extra(30000, 2, seed=91),
    lambda: gen.random_extra(1500, 2, seed=92),
    lambda: gen.grid_nd((150, 150), "5"),
    lambda: gen.grid_nd((36, 36), "5"),
]


def test_calls_of_different_sizes_at_once():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ts = [f() for f in SIZES]
    errors, first = [], [None] * len(ts)

    def work(k):
        try:
            with Context(0) as c:
                m = c.load_rowptr(*ts[k][1:])
                for i in range(150):
                    res = c.factor(m, l_row_stats=(i % 3 == 2))
                    rc = res.row_counts()["nnz_u_row"]
                    if first[k] is None:
                        first[k] = rc
                    np.testing.assert_array_equal(rc, first[k])
                    res.close()
                m.close()
        except Exception as e:  # noqa: BLE001
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k % len(ts),)) for k in range(2 * len(ts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
