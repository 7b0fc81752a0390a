"""Chains of short products, each of the one before: the single-CTA product may
be resident before the kernel that writes its operands has ended."""
import re
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

CSRC = Path(__file__).resolve().parent.parent / "simd_bigint_b200" / "csrc"


def test_operands_are_not_read_through_the_read_only_path():
    """ld.global.nc wants memory that nothing writes while the kernel lives."""
    src = re.sub(r"//[^\n]*", "", (CSRC / "sbg_school.cu").read_text())
    body = src[src.index(" k_school("):src.index(" k_school_b(")]
    assert "pdl_enter()" in body and "__ldg(" not in body


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 20])
def test_chain(ctx, n):
    """r_k = r_(k-1) * a_k, results and factors side by side in one buffer."""
    import torch
    rng = np.random.default_rng(n)
    steps = (128 - n) // n
    parts, at = [rand_limbs(n, rng)], [0]
    for k in range(1, steps + 1):
        parts += [rand_limbs(n, rng), np.zeros((k + 1) * n, dtype=np.uint64)]
    for p in parts:
        at.append(at[-1] + len(p))
    x = torch.from_numpy(np.concatenate(parts).view(np.int64)).cuda()
    torch.cuda.synchronize()
    view = lambda i: x[at[i]:at[i + 1]]  # noqa: E731
    for _ in range(3):
        for k in range(1, steps + 1):
            ctx.mul(view(2 * k), view(0 if k == 1 else 2 * k - 2), view(2 * k - 1))
    ctx.sync()
    want = parts[0]
    for k in range(1, steps + 1):
        want = O.school_mul(want, parts[2 * k - 1])
        assert np.array_equal(view(2 * k).cpu().numpy().view(np.uint64), want), k
