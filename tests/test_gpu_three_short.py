"""The transform lengths 3 * 2^12 .. 3 * 2^15: products, squares and middle
products at both ends of each class, alone, in a batch and as the wrapped
products of a division."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _np(t):
    return t.cpu().numpy().view(np.uint64)


def _shapes():
    out = []
    for k in range(12, 16):
        lo, hi = (1 << (k + 1)) + 1, 3 << k            # an + bn - 1
        out += [(lo // 2 + 1, (lo + 1) // 2), (lo - 5, 6), (hi // 2 + 1, hi // 2), (hi + 1 - (1 << k), 1 << k),
                (hi, 1), (hi // 2 + 1, hi // 2 + 1)]    # the last one is just beyond
    return out


@pytest.mark.parametrize("an,bn", _shapes())
def test_products(ctx, an, bn):
    import torch
    rng = np.random.default_rng(an * 3 + bn)
    for a, b in ((rand_limbs(an, rng), rand_limbs(bn, rng)),
                 (np.full(an, 2**64 - 1, dtype=np.uint64), np.full(bn, 2**64 - 1, dtype=np.uint64))):
        r = torch.empty(an + bn, dtype=torch.int64, device="cuda")
        ta, tb = _dev(a), _dev(b)
        ctx.mul(r, ta, tb)
        ctx.sync()
        assert np.array_equal(_np(r), O.port_mul(a, b))


@pytest.mark.parametrize("k", [12, 13, 14, 15])
def test_squares_and_middle_products(ctx, k):
    import torch
    rng = np.random.default_rng(k)
    for n in ((1 << k) + 1, 3 << (k - 1)):
        a = rand_limbs(n, rng)
        r = torch.empty(2 * n, dtype=torch.int64, device="cuda")
        ta = _dev(a)
        ctx.sqr(r, ta)
        ctx.sync()
        assert np.array_equal(_np(r), O.port_mul(a, a))
    an, bn = (3 << k) - 1, 1 << k
    a, b = rand_limbs(an, rng), rand_limbs(bn, rng)
    r = torch.empty(an - bn + 3, dtype=torch.int64, device="cuda")
    ta, tb = _dev(a), _dev(b)
    ctx.mulmid(r, ta, tb)
    ctx.sync()
    assert np.array_equal(_np(r), O.mulmid(a, b, "ntt"))


@pytest.mark.parametrize("engine", [0, 1, 2])
def test_batch(ctx, engine):
    import torch
    import simd_bigint_b200 as sbg
    rng = np.random.default_rng(77)
    keep, jobs = [], []
    for i, (an, bn) in enumerate(_shapes() + [(5000, 5000), (20000, 3000)]):
        a = rand_limbs(an, rng)
        b = a if i % 4 == 3 else rand_limbs(bn, rng)
        kind = sbg.JOB_SQR if i % 4 == 3 else sbg.JOB_MUL
        ta, tb = _dev(a), _dev(b)
        r = torch.empty(len(a) + len(b), dtype=torch.int64, device="cuda")
        keep.append((a, b, ta, tb, r))
        jobs.append((kind, r.data_ptr(), ta.data_ptr(), tb.data_ptr(), len(a), len(b)))
    torch.cuda.synchronize()
    bt = sbg.Batch(ctx, jobs)
    bt.set_engine(engine)
    bt.capture()
    for _ in range(2):
        bt.run()
    ctx.sync()
    bt.close()
    for a, b, _, _, r in keep:
        assert np.array_equal(_np(r), O.port_mul(a, b)), (len(a), len(b))


@pytest.mark.parametrize("n", [9000, 11000, 17000, 23000])
def test_divisions(ctx, n):
    import torch
    rng = np.random.default_rng(n)
    num, d = rand_limbs(2 * n, rng), rand_limbs(n, rng)
    d[-1] |= np.uint64(1 << 63)
    q = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    r = torch.empty(n, dtype=torch.int64, device="cuda")
    tn, td = _dev(num), _dev(d)
    ctx.divrem(q, r, tn, td)
    i = lambda x: int.from_bytes(np.ascontiguousarray(x, dtype="<u8").tobytes(), "little")  # noqa: E731
    wq, wr = divmod(i(num), i(d))
    assert i(_np(q)) == wq and i(_np(r)) == wr
