"""The request loop's routes: symmetric requests by the chain, the others by the
hubs' launch in a lane, what that leaves by traverse_kernel, side by side; few
CTAs; budgets that were enough for traverse_kernel's workspace alone, where the
chain's makes room."""
import threading
import time

import numpy as np
import pytest

from gsofatpds_b200 import _lib as C
from gsofatpds_b200 import Context, GsofaError, gen
from tests.helpers import scrambled_csr
from tests.test_gpu_serving import _alone, _cuda, _same, _submit

pytestmark = pytest.mark.gpu

MESH = gen.grid_nd((60, 50), "9")[1:]
CORE = gen.circuit_like(6000, target_nnz=52000, seed=81)[1:]
BAND = gen.random_banded(7000, bw=3, extra=0, seed=82)[1:]
ROWS = gen.grid_nd((14, 14, 14), "27")[1:]
SPECS = [MESH, CORE, BAND, ROWS]


@pytest.fixture(scope="module")
def ctx():
    _cuda()
    with Context(0) as c:
        yield c


@pytest.fixture(scope="module")
def refs(ctx):
    return [_alone(ctx, s) for s in SPECS]


def serve(srv, refs, order, pause=0.0):
    tickets = []
    for k in order:
        tickets.append((k, _submit(srv, SPECS[k])))
        if pause:
            time.sleep(pause)
    for k, t in tickets:
        got = srv.wait(t, 60000)
        assert got is not None, "request of kind %d timed out" % k
        _same("kind %d" % k, got, refs[k])
        got.close()


@pytest.mark.parametrize("ctas", [0, 1, 2, 5, 40])
@pytest.mark.parametrize("block", [0, 1024])
def test_both_kinds_with_few_ctas(ctx, refs, ctas, block):
    with ctx.server(max_n=8000, sources_in_flight=ctas, threads_per_source=block) as srv:
        serve(srv, refs, [0, 1, 2, 3, 0, 1])
        serve(srv, refs, [1, 1, 2])
        serve(srv, refs, [0, 3, 0])
        serve(srv, refs, [3, 2, 0, 1], pause=0.004)


def test_neither_kind_waits_for_the_other(ctx, refs):
    """While one kind keeps coming, requests of the other are served."""
    with ctx.server(max_n=8000) as srv:
        stop = threading.Event()
        done = [0]

        def flood():
            while not stop.is_set():
                ts = [_submit(srv, ROWS) for _ in range(6)]
                for t in ts:
                    srv.wait(t, 60000).close()
                done[0] += 6

        th = threading.Thread(target=flood)
        th.start()
        try:
            for k in (1, 2, 1, 2):
                serve(srv, refs, [k])
        finally:
            stop.set()
            th.join()
        assert done[0] > 0


def test_every_route(ctx):
    """Unsymmetric requests of a lane's own making: few rows, entries twice, a
    malformed one, none at all; beside symmetric ones."""
    rng = np.random.default_rng(84)
    few = gen.random_extra(700, 2, seed=85)[1:]
    _, rp, col = gen.random_extra(2000, 3, seed=86)
    twice = scrambled_csr(rng, [set(col[rp[v]:rp[v + 1]]) for v in range(2000)], dup_prob=0.3)
    one = gen.from_coo(1, [0], [0])[1:]
    large = gen.random_banded(90000, bw=6, extra=2, seed=87)[1:]
    specs = [few, twice, one, MESH, BAND, large]
    want = [_alone(ctx, x) for x in specs]
    bad = col.copy()
    bad[11] = 1 << 30
    with ctx.server(max_n=100000) as srv:
        for _ in range(2):
            tickets = [_submit(srv, x) for x in specs]
            t_bad = srv.submit_rowptr(rp, bad)
            t_none = srv.submit_rowptr(np.zeros(1, np.int64), np.zeros(0, np.int32))
            for t, w in zip(tickets, want):
                got = srv.wait(t, 60000)
                _same("route", got, w)
                got.close()
            with pytest.raises(GsofaError) as e:
                srv.wait(t_bad, 60000)
            assert e.value.status == C.ERR_ARG
            got = srv.wait(t_none, 60000)
            assert got.counts["nnz_u"] == 0
            got.close()


def workspaces(ctx, max_n, spec):
    """Bytes of the loop with traverse_kernel alone and with both, and a
    request's footprint."""
    with ctx.server(max_n=max_n, chain=False) as srv:
        least = srv.stats()["fixed_bytes"]
    with ctx.server(max_n=max_n) as srv:
        both = srv.stats()["fixed_bytes"]
        t = _submit(srv, spec)
        srv.wait(t, 60000).close()
        footprint = srv.info(t)["footprint_bytes"]
    return least, both, footprint


@pytest.mark.parametrize("kind", [0, 1])
def test_budget_of_one_kernel(ctx, refs, kind):
    least, both, footprint = workspaces(ctx, 8000, SPECS[kind])
    assert both > least
    with ctx.server(max_n=8000, budget_bytes=least + footprint) as srv:
        serve(srv, refs, [kind, kind])


def test_a_request_that_needs_the_chains_room(ctx, refs):
    big = gen.random_banded(200000, bw=14, extra=4, seed=83)[1:]
    want = _alone(ctx, big)
    least, both, footprint = workspaces(ctx, 200000, big)
    room = max(footprint, both - least) + (8 << 20)
    with ctx.server(max_n=200000, budget_bytes=least + room) as srv:
        first = srv.stats()["fixed_bytes"]
        serve(srv, refs, [0, 1])
        t = _submit(srv, big)
        later = [_submit(srv, SPECS[k]) for k in (0, 1)]
        got = srv.wait(t, 60000)
        _same("large", got, want)
        got.close()
        for k, x in zip((0, 1), later):
            got = srv.wait(x, 60000)
            _same("after", got, refs[k])
            got.close()
        assert first == both and srv.stats()["fixed_bytes"] == least
        serve(srv, refs, [0, 3, 2])


def test_a_context_without_room_for_both(ctx, refs):
    """The context's budget, not the loop's: the chain's workspace goes when a
    request cannot be allocated beside it."""
    big = gen.random_banded(200000, bw=14, extra=4, seed=83)[1:]
    want = _alone(ctx, big)
    least, both, footprint = workspaces(ctx, 200000, big)
    room = max(footprint, both - least) + (8 << 20)
    with Context(0, budget_bytes=least + room) as small:
        with small.server(max_n=200000) as srv:
            assert srv.stats()["fixed_bytes"] == both
            serve(srv, refs, [0, 1])
            t = _submit(srv, big)
            got = srv.wait(t, 60000)
            _same("large", got, want)
            got.close()
            serve(srv, refs, [0, 1])
            assert srv.stats()["fixed_bytes"] == least
