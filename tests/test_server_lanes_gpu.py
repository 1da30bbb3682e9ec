"""The server's two lanes: what holds up the bulk lane's control thread (here an
allocation for which the driver has to map memory) leaves the express lane alone; and
the memory they hand out by themselves, when it is held beyond their share and when it
is in pieces."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bytes(pa, q):
    """What a request with CSR outputs is admitted against."""
    sizes = [ctypes.c_uint64() for _ in range(3)]
    pa.check(pa.lib().pa_csr_bytes(ctypes.byref(q), *map(ctypes.byref, sizes)), "pa_csr_bytes")
    return sum(pa.sizes(q)) + sum(x.value for x in sizes)


def test_bulk_allocation_does_not_hold_up_express_requests(pa, cuda_ok):
    budget = 64 << 30
    if torch.cuda.mem_get_info()[0] < 2 * budget:
        pytest.skip("needs 128 GB of free device memory")
    # fits the budget, but not the bulk lane's share of it (7/8): its pool has to grow
    big = pa.make_params(60_000_000, 32, 0.9, seed=1)
    while _bytes(pa, big) < 0.95 * budget:
        big.n += 1_000_000
    small = [pa.make_params(5000 + i, 4, 0.5, seed=i) for i in range(400)]
    # every request may be in flight at once: one that waits does so for the thread
    with pa.Server(budget_bytes=budget, outputs=pa.PA_OUT_CSR, max_inflight=1000) as srv:
        for q in small[:5]:
            t = srv.submit(q)
            srv.wait(t)
            srv.release(t)
        waits = []
        tickets = []
        bulk = None
        for i, q in enumerate(small):
            tickets.append(srv.submit(q))
            if i == 50:
                bulk = srv.submit(big)
            time.sleep(0.0005)
        for t in tickets:
            rc, res = srv.wait(t)
            assert rc == 0 and res.status == 0
            waits.append((res.t_start_ns - res.t_submit_ns) / 1e6)
            srv.release(t)
        rc, res = srv.wait(bulk)
        assert rc == 0 and res.status == 0
        srv.release(bulk)
    # a pool grows at some 5 ms a GB, and it has to by 5 GB at least; admission itself
    # takes a control loop's turn, well under a millisecond
    assert max(waits) < 10.0, max(waits)


def test_large_request_among_held_results(pa, cuda_ok):
    """A request larger than any piece of memory between the results that a client
    holds: the free pieces are moved together, the device's other memory is left alone,
    and the held results stay what they were."""
    budget = 2 << 30
    held = [pa.make_params(1_000_000 + 1000 * i, 7, 0.5, seed=i, id_bits=32) for i in range(28)]
    large = pa.make_params(10_000_001, 8, 0.5, seed=99, id_bits=32)
    whole = pa.make_params(20_000_003, 8, 0.5, seed=7, id_bits=32)
    # what the reference generation and the comparison load and keep is not the server's
    want, _ = pa.generate(large)
    assert torch.equal(want, want.clone())
    del want
    # express_edges = 1: all of them in one lane
    with pa.Server(budget_bytes=budget, express_edges=1) as srv:
        tickets = [srv.submit(q) for q in held]
        for t in tickets:
            rc, res = srv.wait(t)
            assert rc == 0 and res.status == 0
        torch.cuda.empty_cache()
        free_before = torch.cuda.mem_get_info()[0]
        for turn in range(3):
            for t in tickets[1::2]:
                assert srv.release(t) == 0
            t = srv.submit(large)
            rc, res = srv.wait(t)
            assert rc == 0 and res.status == 0
            want, _ = pa.generate(large)
            assert torch.equal(pa.Server.edges_view(res, 32), want)
            del want
            assert srv.release(t) == 0
            for i, (t, q) in enumerate(zip(tickets, held)):
                if i % 2 == 0:
                    rc, res = srv.poll(t)
                    want, _ = pa.generate(q)
                    assert torch.equal(pa.Server.edges_view(res, 32), want)
            del want
            tickets[1::2] = [srv.submit(q) for q in held[1::2]]
            for t in tickets[1::2]:
                rc, res = srv.wait(t)
                assert rc == 0 and res.status == 0
        torch.cuda.empty_cache()
        assert free_before - torch.cuda.mem_get_info()[0] < (64 << 20)
        for t in tickets:
            assert srv.release(t) == 0
        t = srv.submit(whole)
        rc, res = srv.wait(t)
        assert rc == 0 and res.status == 0
        want, _ = pa.generate(whole)
        assert torch.equal(pa.Server.edges_view(res, 32), want)
        assert srv.release(t) == 0


def test_express_results_held_beyond_the_lanes_share(pa, cuda_ok):
    """Results of small requests that together outgrow the express lane's range are
    served from its pool, and released ones make room again; all as generated alone."""
    with pa.Server(budget_bytes=512 << 20, outputs=pa.PA_OUT_PAIRS | pa.PA_OUT_CSR) as srv:
        for turn in range(3):
            prms = [pa.make_params(20_000 + 997 * i, 1 + i % 9, 0.4, seed=100 * turn + i,
                                   id_bits=32 if i % 3 else 64) for i in range(60)]
            total = sum(_bytes(pa, q) for q in prms)
            assert (512 << 20) / 8 < total < (512 << 20)
            tickets = [srv.submit(q) for q in prms]
            order = list(range(60))
            for i in order:
                rc, res = srv.wait(tickets[i])
                assert rc == 0 and res.status == 0
            for i in order[::2] + order[1::2]:
                rc, res = srv.poll(tickets[i])
                want, _ = pa.generate(prms[i])
                assert torch.equal(pa.Server.edges_view(res, prms[i].id_bits), want)
                rp, col = pa.Server.csr_view(res, prms[i].n, prms[i].id_bits)
                want_rp, want_col = pa.build_csr(prms[i], want)
                assert torch.equal(rp, want_rp) and torch.equal(col, want_col)
                assert srv.release(tickets[i]) == 0
        deadline = time.time() + 5
        while srv.stats().bytes_in_use and time.time() < deadline:
            time.sleep(0.01)
        st = srv.stats()
        assert st.bytes_in_use == 0 and st.failed == 0 and st.released == 180
