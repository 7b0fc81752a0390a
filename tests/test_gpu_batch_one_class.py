"""Batches whose jobs all have one transform length: nothing runs beside their
launches, which may then overlap (dependent launches, in a captured graph too)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


# (an, bn, jobs, launches a run): the schoolbook class, each kernel of the
# transform classes, row launches of at most one CTA per SM and of more, and one
# beyond the dependent launches' 2^20 points
CASES = [(30, 20, 5, 1), (100, 100, 3, 1), (700, 600, 40, 1), (2000, 1500, 7, 1), (4000, 4000, 2, 4), (4000, 4000, 20, 4),
         (6000, 6000, 3, 4), (9000, 9000, 9, 4), (40000, 50000, 2, 4), (33000, 33000, 1, 4), (100000, 110000, 4, 4),
         (700000, 400000, 1, 4)]


@pytest.mark.parametrize("an,bn,count,launches", CASES)
def test_captured_and_replayed(ctx, an, bn, count, launches):
    import torch
    import simd_bigint_b200 as sbg
    rng = np.random.default_rng(an + count)
    ta = [torch.zeros(an, dtype=torch.int64, device="cuda") for _ in range(count)]
    tb = [torch.zeros(bn, dtype=torch.int64, device="cuda") for _ in range(count)]
    r = [torch.zeros(an + bn, dtype=torch.int64, device="cuda") for _ in range(count)]
    torch.cuda.synchronize()
    bt = sbg.Batch(ctx, [(sbg.JOB_MUL, z.data_ptr(), x.data_ptr(), y.data_ptr(), an, bn) for x, y, z in zip(ta, tb, r)])
    try:
        for form in ("launched", "captured", "replayed"):
            hosts = [(rand_limbs(an, rng), rand_limbs(bn, rng)) for _ in range(count)]
            for (a, b), x, y in zip(hosts, ta, tb):
                x.copy_(_dev(a))
                y.copy_(_dev(b))
            torch.cuda.synchronize()
            if form == "captured":
                bt.capture()
            before = ctx.launches()
            for _ in range(3):                   # back to back: each run over the one before
                bt.run()
            assert ctx.launches() - before == 3 * launches
            ctx.sync()
            for (a, b), z in zip(hosts, r):
                assert np.array_equal(z.cpu().numpy().view(np.uint64), O.port_mul(a, b)), form
    finally:
        bt.close()
