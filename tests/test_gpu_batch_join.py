"""Batches in which a few short jobs of 3 * 2^k points join the class of 2^(k+2)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


# (3 * 2^k jobs, with a 2^(k+2) job beside them, launches a run): 2^17 points is the line
@pytest.mark.parametrize("k,count,beside,launches", [(12, 1, True, 4), (12, 10, True, 4), (12, 11, True, 8), (12, 2, False, 4),
                                                     (13, 5, True, 4), (13, 6, True, 8), (14, 2, True, 4), (14, 3, True, 8),
                                                     (15, 1, True, 4), (15, 2, True, 8)])
def test_jobs(ctx, k, count, beside, launches):
    import torch
    import simd_bigint_b200 as sbg
    rng = np.random.default_rng(10 * k + count)
    top = 3 << k
    shapes = [(sbg.JOB_MUL, top // 2 + 1, top // 2), (sbg.JOB_MUL, top, 1), (sbg.JOB_SQR, top // 2, 0),
              (sbg.JOB_MULMID, top, 1 + top // 3), (sbg.JOB_MUL, (1 << (k + 1)) + 1, 1)]
    keep, jobs = [], []
    for kind, an, bn in [shapes[i % 5] for i in range(count)] + [(sbg.JOB_MUL, 1 << (k + 1), 1 << (k + 1))] * beside:
        a = rand_limbs(an, rng)
        b = a if kind == sbg.JOB_SQR else rand_limbs(bn, rng)
        ta, tb = _dev(a), _dev(b)
        r = torch.empty(sbg.out_limbs(kind, an, bn), dtype=torch.int64, device="cuda")
        want = O.mulmid(a, b, "ntt") if kind == sbg.JOB_MULMID else O.port_mul(a, b)
        keep.append((ta, tb, r, want))
        jobs.append((kind, r.data_ptr(), ta.data_ptr(), tb.data_ptr(), an, bn))
    torch.cuda.synchronize()
    bt = sbg.Batch(ctx, jobs)
    before = ctx.launches()
    bt.run()
    ctx.sync()
    assert ctx.launches() - before == launches
    bt.close()
    for form in ("planned", "list"):
        if form == "list":
            arr = (sbg.Job * len(jobs))()
            for i, (kind, r, a, b, an, bn) in enumerate(jobs):
                arr[i].kind, arr[i].rp, arr[i].ap, arr[i].bp, arr[i].an, arr[i].bn = kind, r, a, b, an, bn
            assert sbg.lib().sbg_mul_batch(ctx.handle, C.addressof(arr), len(jobs)) == 0
        for _, _, r, want in keep:
            assert np.array_equal(r.cpu().numpy().view(np.uint64), want), form
            r.zero_()
        torch.cuda.synchronize()


def test_wrapped_products_keep_their_length(ctx):
    """A division's wrapped product is one modulo B^L - 1: its length stays, with
    a longer class beside it (9000 and 11000 limbs wrap at 3 * 2^12, 13000 at 2^14)."""
    import torch
    rng = np.random.default_rng(3)
    i = lambda x: int.from_bytes(np.ascontiguousarray(x, dtype="<u8").tobytes(), "little")  # noqa: E731
    keep, jobs = [], []
    for n in (9000, 13000, 11000, 20000, 27000):
        x, d = rand_limbs(2 * n, rng), rand_limbs(n, rng)
        d[-1] |= np.uint64(1 << 63)
        tx, td = _dev(x), _dev(d)
        q = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        r = torch.empty(n, dtype=torch.int64, device="cuda")
        keep.append((x, d, tx, td, q, r))
        jobs.append((q.data_ptr(), r.data_ptr(), tx.data_ptr(), td.data_ptr(), 2 * n, n))
    torch.cuda.synchronize()
    ctx.divrem_batch(jobs)
    for x, d, _, _, q, r in keep:
        wq, wr = divmod(i(x), i(d))
        assert i(q.cpu().numpy().view(np.uint64)) == wq and i(r.cpu().numpy().view(np.uint64)) == wr
