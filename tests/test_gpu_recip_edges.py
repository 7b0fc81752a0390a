"""Reciprocals and divisions whose Newton steps leave the settled-by-a-few-
limbs paths: structured divisors (powers of two, all ones, zero tails, sparse)
give zero or all-ones limbs where those paths read them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def _int(x) -> int:
    return int.from_bytes(np.ascontiguousarray(x, dtype="<u8").tobytes(), "little")


def _limbs(v: int, n: int) -> np.ndarray:
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype="<u8").copy()


def _divisors(n: int):
    B = 1 << 64
    top = B**n // 2
    rng = np.random.default_rng(n)
    r = _int(rng.integers(0, 2**64, n, dtype=np.uint64))
    h = n - (n - 1) // 2
    yield "half", top
    yield "half+1", top + 1
    yield "ones", B**n - 1
    yield "ones-1", B**n - 2
    yield "top ones", B**n - B ** (n - h)
    yield "top half, low ones", top + B ** (n - h) - 1
    yield "one limb", top | (B ** (n - 1) * 0x1234567)
    yield "middle", top + B ** (n // 2)
    yield "random top, zero low", (r >> (64 * (n // 3)) << (64 * (n // 3))) | top
    yield "random top, ones low", r | top | (B ** (n // 3) - 1)
    yield "2/3", (2 * B**n) // 3 | top
    yield "random", r | top


# sizes on both sides of every threshold: the base case, one-CTA products,
# four-step lengths, steps on clusters
@pytest.mark.parametrize("n", [128, 129, 255, 400, 1000, 2047, 4097, 6143, 6145, 9000, 13000])
def test_structured_reciprocals(ctx, n):
    import torch
    for name, d in _divisors(n):
        v = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        ctx.recip(v, _dev(_limbs(d, n)))
        want = ((1 << (128 * n)) - 1) // d - (1 << (64 * n))
        assert _int(v.cpu().numpy().view(np.uint64)) == want, (n, name)


@pytest.mark.parametrize("n", [130, 1500, 7000])
def test_structured_divisions(ctx, n):
    import torch
    cases = [(name, d) for name, d in _divisors(n)]
    rng = np.random.default_rng(n + 1)
    jobs, keep = [], []
    for i, (_, d) in enumerate(cases):
        nums = [(1 << (128 * n)) - 1, d * (d - 1), d * d - 1, d * ((1 << (64 * n)) - 1),
                _int(rng.integers(0, 2**64, 2 * n, dtype=np.uint64))]
        x = nums[i % len(nums)]
        tn, td = _dev(_limbs(x, 2 * n)), _dev(_limbs(d, n))
        q = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        r = torch.empty(n, dtype=torch.int64, device="cuda")
        keep.append((x, d, tn, td, q, r))
        jobs.append((q.data_ptr(), r.data_ptr(), tn.data_ptr(), td.data_ptr(), 2 * n, n))
    torch.cuda.synchronize()
    ctx.divrem_batch(jobs)
    for (name, _), (x, d, _, _, q, r) in zip(cases, keep):
        wq, wr = divmod(x, d)
        assert _int(q.cpu().numpy().view(np.uint64)) == wq, name
        assert _int(r.cpu().numpy().view(np.uint64)) == wr, name


@pytest.mark.parametrize("n", [200, 3000, 8000])
def test_results_over_the_numerator(ctx, n):
    """Quotient or remainder written over the numerator, one division's over
    another's, or all apart: the same results."""
    import torch
    rng = np.random.default_rng(n + 7)
    for layout in ("apart", "remainder over own", "quotient over own", "over the other's"):
        nums = [rng.integers(0, 2**64, 2 * n, dtype=np.uint64) for _ in range(2)]
        divs = [rng.integers(0, 2**64, n, dtype=np.uint64) for _ in range(2)]
        for d in divs:
            d[-1] |= np.uint64(1 << 63)
        tn, td = [_dev(x) for x in nums], [_dev(x) for x in divs]
        q = [torch.empty(n + 1, dtype=torch.int64, device="cuda") for _ in range(2)]
        r = [torch.empty(n, dtype=torch.int64, device="cuda") for _ in range(2)]
        for i in range(2):
            if layout == "remainder over own":
                r[i] = tn[i][:n]
            elif layout == "quotient over own":
                q[i] = tn[i][: n + 1]
            elif layout == "over the other's":
                r[i] = tn[1 - i][n:]
        torch.cuda.synchronize()
        ctx.divrem_batch([(q[i].data_ptr(), r[i].data_ptr(), tn[i].data_ptr(), td[i].data_ptr(), 2 * n, n)
                          for i in range(2)])
        for i in range(2):
            wq, wr = divmod(_int(nums[i]), _int(divs[i]))
            assert _int(q[i].cpu().numpy().view(np.uint64)) == wq, layout
            assert _int(r[i].cpu().numpy().view(np.uint64)) == wr, layout
