"""Full-size parity of the default calls, which are counted on hubs and by the
chain (without per-row L statistics): the same committed oracle answers as
test_gpu_fullsize, every per-row array but the two of the L rows.

  c1, c2, c3  plain calls; c2 also with labels and bitmaps in global memory
  c4          the 512-matrix mix: the graph-captured batch, run twice, and
              every matrix alone
  c5          the 48-request serving stream, all requests in one request loop
"""
import pytest

from gsofatpds_b200 import gen
from tests import fullsize as F
from tests.test_gpu_fullsize import ctx, fixture  # noqa: F401

pytestmark = pytest.mark.gpu


def plain(ctx, t, mss, **kw):  # noqa: F811
    m = ctx.load_rowptr(*t[1:])
    res = ctx.factor(m, max_supernode_size=mss, **kw)
    rec = F.device_record(res, l_rows=False)
    res.close()
    m.close()
    return rec


def test_c1(ctx):  # noqa: F811
    ref, = fixture("c1")
    F.compare(plain(ctx, gen.random_extra(20000, 3, seed=1), 128), ref, "c1")


@pytest.mark.parametrize("kw", [dict(), dict(global_bitmap=True)], ids=["default", "global"])
def test_c2(ctx, kw):  # noqa: F811
    ref, = fixture("c2")
    F.compare(plain(ctx, gen.circuit_like(), 128, **kw), ref, "c2")


def test_c3(ctx):  # noqa: F811
    ref, = fixture("c3")
    F.compare(plain(ctx, gen.grid_nd((64, 64, 64), "7"), 256), ref, "c3")


def test_c4(ctx):  # noqa: F811
    refs = fixture("c4")
    mats = [ctx.load_rowptr(rp, col) for (_, rp, col) in gen.batch_mix(512)]
    b = ctx.batch(mats, max_supernode_size=128)
    for run in range(2):
        b.run()
        for i, ref in enumerate(refs):
            F.compare(F.device_record(b.result(i), l_rows=False), ref, "c4 batch %d run %d" % (i, run))
    b.close()
    for i, (m, ref) in enumerate(zip(mats, refs)):
        res = ctx.factor(m, max_supernode_size=128)
        F.compare(F.device_record(res, l_rows=False), ref, "c4 alone %d" % i)
        res.close()
        m.close()


def test_c5(ctx):  # noqa: F811
    refs = fixture("c5")
    reqs = [gen.make_request(kind, spec) for (_, kind, spec) in gen.request_stream(**gen.SERVE_STREAM)]
    with ctx.server(max(n for (n, _, _) in reqs), max_supernode_size=128) as srv:
        tickets = [srv.submit_rowptr(rp, col) for (_, rp, col) in reqs]
        for k, (t, ref) in enumerate(zip(tickets, refs)):
            res = srv.wait(t, timeout_ms=600000)
            assert res is not None, "request %d timed out" % k
            F.compare(F.device_record(res, l_rows=False), ref, "c5 request %d" % k)
            res.close()
