"""Divisions and reciprocals whose results lie over their own divisor, whole or
in part, or over another division's: the same results as apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _int(x) -> int:
    return int.from_bytes(np.ascontiguousarray(x, dtype="<u8").tobytes(), "little")


def _host(t) -> int:
    return _int(t.cpu().numpy().view(np.uint64))


def _limbs(v: int, n: int) -> np.ndarray:
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype="<u8").copy()


# one-CTA linear steps of one tile and of several, steps on clusters
@pytest.mark.parametrize("n", [128, 200, 3000, 9000, 40000])
@pytest.mark.parametrize("layout", ["remainder", "remainder, shifted up", "remainder, shifted down", "quotient",
                                    "the other's"])
def test_results_over_the_divisor(ctx, n, layout):
    import torch
    rng = np.random.default_rng(n)
    divs, nums = [], []
    for i in range(6):
        d = rng.integers(0, 2**64, n, dtype=np.uint64)
        d[-1] |= np.uint64(1 << 63)
        if i % 2:                                # minimal divisors and full numerators: the most corrections
            d[:] = 0
            d[-1] = np.uint64(1 << 63)
            d[: n // 3] = np.uint64(2**64 - 1)
        x = rng.integers(0, 2**64, 2 * n, dtype=np.uint64) if i % 3 else np.full(2 * n, 2**64 - 1, dtype=np.uint64)
        divs.append(d)
        nums.append(x)
    pad = 33
    bufs = [torch.zeros(n + 2 * pad, dtype=torch.int64, device="cuda") for _ in divs]
    q = [torch.empty(n + 1, dtype=torch.int64, device="cuda") for _ in divs]
    r = [torch.empty(n, dtype=torch.int64, device="cuda") for _ in divs]
    td, tn = [], [_dev(x) for x in nums]
    for i, d in enumerate(divs):
        bufs[i][pad:pad + n] = _dev(d)
        td.append(bufs[i][pad:pad + n])
    for i in range(len(divs)):
        if layout == "remainder":
            r[i] = td[i]
        elif layout == "remainder, shifted up":
            r[i] = bufs[i][2 * pad:2 * pad + n]
        elif layout == "remainder, shifted down":
            r[i] = bufs[i][:n]
        elif layout == "quotient":
            q[i] = bufs[i][pad:pad + n + 1]
        else:
            r[i] = td[i ^ 1]
    torch.cuda.synchronize()
    ctx.divrem_batch([(q[i].data_ptr(), r[i].data_ptr(), tn[i].data_ptr(), td[i].data_ptr(), 2 * n, n)
                      for i in range(len(divs))])
    for i in range(len(divs)):
        wq, wr = divmod(_int(nums[i]), _int(divs[i]))
        assert _host(q[i]) == wq and _host(r[i]) == wr, i


@pytest.mark.parametrize("n", [100, 128, 700, 6200, 9000, 40000])
def test_reciprocals_in_place(ctx, n):
    import torch
    B = 1 << 64
    rng = np.random.default_rng(n + 3)
    r = _int(rng.integers(0, 2**64, n, dtype=np.uint64))
    # divisors whose reciprocal ends in zeros or ones, and a random one
    for d in (B**n // 2, B**n // 2 + 1, B**n - 1, r | B**n // 2, (2 * B**n) // 3 | B**n // 2):
        for shift in (0, 17):
            buf = torch.zeros(n + 17, dtype=torch.int64, device="cuda")
            buf[:n] = _dev(_limbs(d, n))
            v = buf[shift:shift + n]
            torch.cuda.synchronize()
            ctx.recip(v, buf[:n])
            assert _host(v) == ((1 << (128 * n)) - 1) // d - (1 << (64 * n)), shift
