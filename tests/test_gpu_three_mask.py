"""A mask of 0 keeps every transform length a power of two, the short ones too."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


@pytest.mark.parametrize("mask,launches", [(0, 1), (0x00EF0000, 17)])
def test_batch_launches_of_the_queue_engine(ctx, mask, launches):
    import torch
    import simd_bigint_b200 as sbg
    rng = np.random.default_rng(mask + 5)
    keep, jobs = [], []
    # schoolbook, one-CTA and four-step powers of two, and one of each 3 * 2^k, k = 12 .. 15
    for an, bn in [(40, 60), (700, 600), (4000, 3000)] + [(3 << (k - 1), 3 << (k - 1)) for k in range(12, 16)]:
        a, b = rand_limbs(an, rng), rand_limbs(bn, rng)
        ta, tb = _dev(a), _dev(b)
        r = torch.empty(an + bn, dtype=torch.int64, device="cuda")
        keep.append((a, b, ta, tb, r))
        jobs.append((sbg.JOB_MUL, r.data_ptr(), ta.data_ptr(), tb.data_ptr(), an, bn))
    torch.cuda.synchronize()
    old = ctx.len3_mask
    try:
        ctx.set_len3_mask(mask)
        bt = sbg.Batch(ctx, jobs)
        bt.set_engine(0)
        before = ctx.launches()
        bt.run()
        ctx.sync()
        assert ctx.launches() - before == launches
        bt.close()
        for a, b, ta, tb, r in keep:
            want = O.port_mul(a, b)
            assert np.array_equal(r.cpu().numpy().view(np.uint64), want)
            r.zero_()
            torch.cuda.synchronize()
            ctx.mul(r, ta, tb)
            ctx.sync()
            assert np.array_equal(r.cpu().numpy().view(np.uint64), want)
    finally:
        ctx.set_len3_mask(old)
