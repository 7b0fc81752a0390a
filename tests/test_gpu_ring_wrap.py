"""Batched divisions and reciprocals whose descriptor rings wrap inside one call
(rings made small by the test hook), as those of very long batches do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _int(x) -> int:
    return int.from_bytes(np.ascontiguousarray(x, dtype="<u8").tobytes(), "little")


@pytest.fixture()
def small_rings():
    import simd_bigint_b200 as sbg
    L = sbg.lib()
    L.sbg_debug_ring_bytes(256)
    yield sbg
    L.sbg_debug_ring_bytes(0)


def test_division_batches(small_rings):
    import torch
    sbg = small_rings
    rng = np.random.default_rng(31)
    ctx = sbg.Context(0)
    try:
        # first calls small: the rings hold four of their blocks, so the longer
        # ones wrap and grow them in mid-call
        for count in (2, 12, 48, 48, 30):
            jobs, keep = [], []
            for i in range(count):
                n = int(rng.integers(128, 1500))
                nn = 2 * n if i % 3 else n + n // 2
                x, d = rng.integers(0, 2**64, nn, dtype=np.uint64), rng.integers(0, 2**64, n, dtype=np.uint64)
                d[-1] |= np.uint64(1 << 63)
                tx, td = _dev(x), _dev(d)
                q = torch.empty(nn - n + 1, dtype=torch.int64, device="cuda")
                r = torch.empty(n, dtype=torch.int64, device="cuda")
                keep.append((x, d, tx, td, q, r))
                jobs.append((q.data_ptr(), r.data_ptr(), tx.data_ptr(), td.data_ptr(), nn, n))
            torch.cuda.synchronize()
            ctx.divrem_batch(jobs)
            for x, d, _, _, q, r in keep:
                wq, wr = divmod(_int(x), _int(d))
                assert _int(q.cpu().numpy().view(np.uint64)) == wq, (count, len(x), len(d))
                assert _int(r.cpu().numpy().view(np.uint64)) == wr, (count, len(x), len(d))
    finally:
        ctx.close()


def test_batched_reciprocals(small_rings, ctx):
    import torch
    sbg = small_rings
    rng = np.random.default_rng(32)
    srv = sbg.Server(ctx, arena_bytes=1 << 30, slots=2, max_batch=64, recip_workers=1)
    try:
        divs = []
        for _ in range(120):
            d = rng.integers(0, 2**64, int(rng.integers(128, 1200)), dtype=np.uint64)
            d[-1] |= np.uint64(1 << 63)
            divs.append((d, _dev(d)))
        torch.cuda.synchronize()
        tickets = srv.submit_many([(2, t.data_ptr(), len(d), 0, 0) for d, t in divs])
        want = dict(zip(tickets, divs))
        for _ in range(60):
            if not want:
                break
            for ticket, status, rp, rn, *_ in srv.poll_detail(wait_ms=1000):
                assert status == 0
                d, _ = want.pop(ticket)
                v = _int(srv.result(rp, rn).cpu().numpy().view(np.uint64))
                n = len(d)
                assert v == ((1 << (128 * n)) - 1) // _int(d) - (1 << (64 * n)), n
                srv.release(ticket)
        assert not want
    finally:
        srv.close()
