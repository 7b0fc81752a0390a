"""Products of 2^8 .. 2^12 transform points: the one-launch cluster kernel, at
the edges of its lengths, of its carry runs and of its operand shapes."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _mul(ctx, a, b):
    import torch
    r = torch.full((len(a) + len(b),), -1, dtype=torch.int64, device="cuda")
    ta, tb = _dev(a), _dev(b)
    ctx.mul(r, ta, tb)
    ctx.sync()
    return r.cpu().numpy().view(np.uint64)


# totals around every power of two (an + bn - 1 coefficients) and around the
# multiples of five runs of limbs
TOTALS = sorted({t + d for t in (129, 257, 513, 1025, 2049, 4097) for d in (-1, 0, 1) if 129 <= t + d <= 4097}
                | {200, 640, 1000, 3199, 3201, 4090})


@pytest.mark.parametrize("total", TOTALS)
def test_products_at_the_edges(ctx, total):
    rng = np.random.default_rng(total)
    for an in sorted({total // 2, total - 1, total - 2, (2 * total) // 3}):
        a, b = rand_limbs(an, rng), rand_limbs(total - an, rng)
        assert np.array_equal(_mul(ctx, a, b), O.port_mul(a, b)), (an, total - an)


@pytest.mark.parametrize("n", [65, 128, 129, 500, 1024, 1025, 2048])
def test_squares_and_all_ones(ctx, n):
    import torch
    ones = np.full(n, 2**64 - 1, dtype=np.uint64)
    for a in (rand_limbs(n, np.random.default_rng(n)), ones):
        r = torch.empty(2 * n, dtype=torch.int64, device="cuda")
        ta = _dev(a)
        ctx.sqr(r, ta)
        ctx.sync()
        assert np.array_equal(r.cpu().numpy().view(np.uint64), O.port_mul(a, a))
    assert np.array_equal(_mul(ctx, ones, ones), O.port_mul(ones, ones))
    # carries through every limb: (B^n - 1) * 1, and sparse operands
    one = np.zeros(n, dtype=np.uint64)
    one[0] = 1
    one[-1] = 1
    assert np.array_equal(_mul(ctx, ones, one), O.port_mul(ones, one))


@pytest.mark.parametrize("an,bn", [(200, 1), (256, 100), (1024, 1024), (1025, 513), (4096, 1), (4096, 2047), (4096, 4096)])
def test_middle_products(ctx, an, bn):
    import torch
    rng = np.random.default_rng(an * 7 + bn)
    a, b = rand_limbs(an, rng), rand_limbs(bn, rng)
    r = torch.empty(an - bn + 3, dtype=torch.int64, device="cuda")
    ta, tb = _dev(a), _dev(b)
    ctx.mulmid(r, ta, tb)
    ctx.sync()
    assert np.array_equal(r.cpu().numpy().view(np.uint64), O.mulmid(a, b))


def test_corrupted_top_residue_spills(ctx):
    import simd_bigint_b200 as sbg
    L = sbg.lib()
    rng = np.random.default_rng(5)
    a, b = rand_limbs(700, rng), rand_limbs(650, rng)
    try:
        assert L.sbg_debug_inject(sbg.INJECT_TOP) == 0
        with pytest.raises(sbg.SbgError) as e:
            _mul(ctx, a, b)
        assert e.value.status == 6               # SBG_ESPILL
    finally:
        assert L.sbg_debug_inject(0) == 0
    assert np.array_equal(_mul(ctx, a, b), O.port_mul(a, b))
