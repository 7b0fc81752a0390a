"""Divisions, reciprocals and one-job batches work in the product lists' arena:
the workspace of the context's own products is neither needed nor grown."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tests.common import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int64)).cuda()


def test_workspace_is_not_grown():
    import torch
    import simd_bigint_b200 as sbg
    n = 20000
    ctx = sbg.Context(0)
    L = sbg.lib()
    rng = np.random.default_rng(11)
    try:
        # the tables of every length below, without a workspace (a batch each:
        # in one, short lengths join longer ones)
        x = torch.zeros(1 << 17, dtype=torch.int64, device="cuda")
        for ln in [1 << k for k in range(7, 17)] + [3 << k for k in range(12, 15)]:
            sbg.Batch(ctx, [(sbg.JOB_MUL, x.data_ptr(), x.data_ptr(), x.data_ptr(), ln, 1)]).close()
        d = rand_limbs(n, rng)
        d[-1] |= np.uint64(1 << 63)
        a, b = rand_limbs(9000, rng), rand_limbs(8000, rng)
        td, ta, tb = _dev(d), _dev(a), _dev(b)
        v = torch.empty(n, dtype=torch.int64, device="cuda")
        r = torch.empty(17000, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        L.sbg_debug_fail_allocs(1)               # a workspace cannot be had
        ctx.recip(v, td)
        job = sbg.Job(r.data_ptr(), ta.data_ptr(), tb.data_ptr(), 9000, 8000, sbg.JOB_MUL, 0)
        assert L.sbg_mul_batch(ctx.handle, C.addressof(job), 1) == 0
        with pytest.raises(sbg.SbgError):
            ctx.mul(r, ta, tb)                   # which needs one
    finally:
        L.sbg_debug_fail_allocs(0)
        ctx.close()
    dv = int.from_bytes(d.tobytes(), "little")
    assert int.from_bytes(v.cpu().numpy().tobytes(), "little") == ((1 << (128 * n)) - 1) // dv - (1 << (64 * n))
    assert np.array_equal(r.cpu().numpy().view(np.uint64), O.port_mul(a, b))
