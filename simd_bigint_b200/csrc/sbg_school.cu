// sbg_school.cu -- the small-size front end: schoolbook products of at most
// SBG_SCHOOL_MAX output limbs, one warp per product in batches, one CTA for a
// product alone.
//
// Below a few dozen limbs a five-prime transform is all overhead (five CTAs,
// three transforms and a CRT launch for a handful of limbs).  The reference
// covers this band with its own basecase kernels (include/u64cvt.h:100-106:
// an asm basecase up to 6 limbs, include/mul.h:764 basecase / Toom below the
// FFT band); here a warp forms the product column by column in exact 64-bit
// arithmetic:
//   * lane l owns the columns k = 32 s + l (s = 0..3), accumulating
//     sum_{i+j=k} a_i b_j in 192 bits (lo, mid, hi) with the PTX multiply-add
//     carry chain (mad.lo.cc / madc.hi.cc / addc);
//   * limb m of the product is lo_m + mid_{m-1} + hi_{m-2} + carries, the
//     same three-stream recombination as the CRT kernel's; the neighbour
//     terms come by shuffles, the sum carries (0..2) from the lane below, and
//     the ripple carries of a 32-limb step are resolved at once from the
//     lanes' generate / propagate ballots: carries = (p + (g << 1 | c)) ^ p.
// Operands are staged in shared memory (2 KB per warp), so each a_i is a
// broadcast and the b_{k-i} of a warp are 32 consecutive words.
#include <cuda_runtime.h>

#include "sbg_internal.h"
#include "sbg_school.cuh"

namespace sbg {

// One product alone is a chain of latencies, so it is spread over a CTA: warp
// (part, step) accumulates every SCHOOL_PARTS-th term of the 32 columns of its
// step, the parts' sums meet in shared memory and one warp per step resolves
// its limbs.  b sits between zeros, so a lane's terms need no range test.
// 60 x 40 limbs against the one-warp form, which batches keep (there the products
// fill the device): 12.3 -> 4.1 us a call back to back, the host's pace; 6.0 ->
// 2.0 us in a captured chain of them.
#define SCHOOL_PARTS 4
#define SCHOOL_STEPS (SBG_SCHOOL_MAX / 32)
#define SCHOOL_T (32 * SCHOOL_PARTS * SCHOOL_STEPS)
__global__ void __launch_bounds__(SCHOOL_T) k_school(const uint64_t* __restrict__ a, int an,
                                                     const uint64_t* __restrict__ b, int bn,
                                                     uint64_t* __restrict__ out) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int MAX = SBG_SCHOOL_MAX;
    __shared__ uint64_t sa[MAX], sb[3 * MAX];              // b_j at sb[MAX + j]
    __shared__ uint64_t s_lo[SCHOOL_PARTS][MAX], s_mid[SCHOOL_PARTS][MAX];
    __shared__ uint32_t s_hi[SCHOOL_PARTS][MAX];
    __shared__ uint64_t c_lo[MAX + 3], c_mid[MAX + 3];     // column k at k + 3
    __shared__ uint32_t c_hi[MAX + 3], s_g[SCHOOL_STEPS], s_p[SCHOOL_STEPS];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int step = wid % SCHOOL_STEPS, part = wid / SCHOOL_STEPS;
    const int n = an + bn;
    pdl_enter();
    // the kernel before may have written the operands while this one was
    // already resident: not through the read-only path
    for (int i = tid; i < 3 * MAX; i += SCHOOL_T) sb[i] = i >= MAX && i < MAX + bn ? __ldcg(&b[i - MAX]) : 0;
    if (tid < an) sa[tid] = __ldcg(&a[tid]);
    if (tid < 3) {
        c_lo[tid] = c_mid[tid] = 0;
        c_hi[tid] = 0;
    }
    __syncthreads();
    const int k = 32 * step + lane;
    {
        uint64_t lo = 0, mid = 0;
        uint32_t hi = 0;
        // terms that any of the step's columns has
        const int i0 = max(0, 32 * step - bn + 1), i1 = min(32 * step + 31, an - 1);
        const uint64_t* y = sb + MAX + k;
#pragma unroll 4
        for (int i = i0 + part; i <= i1; i += SCHOOL_PARTS) mac192(lo, mid, hi, sa[i], y[-i]);
        s_lo[part][k] = lo;
        s_mid[part][k] = mid;
        s_hi[part][k] = hi;
    }
    __syncthreads();
    uint64_t lo = 0, mid = 0, z = 0;
    uint32_t hi = 0, g = 0, p = 0;
    if (part == 0) {
#pragma unroll
        for (int q = 0; q < SCHOOL_PARTS; ++q) {
            asm("add.cc.u64 %0, %0, %3;\n\t"
                "addc.cc.u64 %1, %1, %4;\n\t"
                "addc.u32 %2, %2, %5;"
                : "+l"(lo), "+l"(mid), "+r"(hi)
                : "l"(s_lo[q][k]), "l"(s_mid[q][k]), "r"(s_hi[q][k]));
        }
        c_lo[k + 3] = lo;
        c_mid[k + 3] = mid;
        c_hi[k + 3] = hi;
    }
    __syncthreads();
    if (part == 0) {
        // limb k: lo_k + mid_{k-1} + hi_{k-2} + the sum carry of limb k-1
        uint64_t y, t;
        uint32_t kk, kb;
        school_sum3(lo, c_mid[k + 2], c_hi[k + 1], y, kk);
        school_sum3(c_lo[k + 2], c_mid[k + 1], c_hi[k], t, kb);
        z = y + kb;
        g = __ballot_sync(FULL, z < y);
        p = __ballot_sync(FULL, z == ~0ull);
        if (lane == 0) {
            s_g[step] = g;
            s_p[step] = p;
        }
    }
    __syncthreads();
    if (part == 0) {
        uint32_t cin = 0;
        for (int q = 0; q < step; ++q)
            cin = (uint32_t)(((uint64_t)s_p[q] + ((s_g[q] << 1) | cin)) >> 32) | (s_g[q] >> 31);
        const uint64_t sum = (uint64_t)p + ((g << 1) | cin);
        if (k < n) out[k] = z + ((((uint32_t)sum ^ p) >> lane) & 1u);
    }
}

// batched: one warp per job (plain products only: cmin = 0, off = 0)
__global__ void __launch_bounds__(32 * SCHOOL_WARPS) k_school_b(const JobDesc* __restrict__ jobs,
                                                                int njobs) {
    __shared__ uint64_t sa[SCHOOL_WARPS][SBG_SCHOOL_MAX], sb[SCHOOL_WARPS][SBG_SCHOOL_MAX];
    const int w = threadIdx.x >> 5;
    const int j = blockIdx.x * SCHOOL_WARPS + w;
    if (j >= njobs) return;
    const JobDesc& J = jobs[j];
    school_warp(J.a, (int)J.an, J.b, (int)J.bn, J.out, sa[w], sb[w]);
}

cudaError_t launch_school(const uint64_t* a, int64_t an, const uint64_t* b, int64_t bn,
                          uint64_t* out, cudaStream_t st) {
    if (an <= 0 || bn <= 0 || an + bn > SBG_SCHOOL_MAX) return cudaErrorInvalidValue;
    return launch_pdl(k_school, true, 1, SCHOOL_T, 0, 1, st, a, (int)an, b, (int)bn, out);
}

cudaError_t launch_school_batch(const JobDesc* djobs, int njobs, cudaStream_t st) {
    if (njobs <= 0) return cudaSuccess;
    k_school_b<<<(njobs + SCHOOL_WARPS - 1) / SCHOOL_WARPS, 32 * SCHOOL_WARPS, 0, st>>>(djobs, njobs);
    return cudaGetLastError();
}

}  // namespace sbg
