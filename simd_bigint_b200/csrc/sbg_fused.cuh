// sbg_fused.cuh -- a whole product of 2^8 <= L <= 2^12 transform points in
// one launch (included by sbg_kernels.cu).
//
// A cluster of five CTAs, one per prime.  Each CTA transforms both operands,
// multiplies and transforms back in shared memory (the operands side by side
// on 256 threads each, radix-16 groups straight from the limbs, the last
// forward pass, the product and the first inverse pass fused in registers;
// twiddles staged in shared memory, since a single product touches each only
// once or twice and would wait for each level's from L2).  The five CTAs
// then read each other's residues through distributed shared memory, rebuild
// the coefficients (two per thread) and resolve the carries: a warp's by
// ballots, the cluster's from the (generate, propagate) bits of all its
// warps.  Nothing goes through global memory between the limbs and the
// product, and no flag is waited for.
// What bounds it is the chain of passes (20,000 clocks at 2^12 points, the
// five SMs issuing 44% of them).  1500 x 1500 limbs, device time a call back
// to back: 30.7 us with the transforms, the flags' memset and the carry scan
// as three launches, 9.4 us.  A batch's classes run it too, one cluster per
// job, with as many threads as the length has radix-16 groups: 128 divisions
// 5.58 -> 5.30 ms, 1024 mixed products 1.352 -> 1.335 ms (640 CTAs of 2^8,
// 2^10 and 2^12 points: 12 to 16, 16 and 40 us against 28, 36 and 67 us with
// one CTA per prime and a carry scan).
// Shorter transforms (2^4 .. 2^7, tiny middle products) keep those launches.
#pragma once

namespace sbg {

#define FU_T 512                               // threads at 2^12 points, and of the row kernel below
// threads at 2^LG points: a radix-16 group of either operand each
__host__ __device__ constexpr int fu_threads(int lg) { return lg <= 9 ? 64 : 1 << (lg - 3); }
#define FU_V 2                                 // limbs per thread in the carry phase

template <int LG>
struct FusedSmem {
    static constexpr int FU_NW = fu_threads(LG) / 32;      // warps
    uint32_t A[padded_len(1 << LG)];
    uint32_t B[padded_len(1 << LG)];
    uint2 twf[1 << LG];
    uint2 twi[1 << LG];
    ulonglong2 xlo[FU_NW][2];              // limbs of each warp's last two lanes
    uint64_t xmid[FU_NW][2];
    uint2 xhi[FU_NW][2];
    uint32_t warp[FU_NW];                  // (G, P) of this CTA's warps
};

__device__ __forceinline__ uint32_t dsmem_ld(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// one middle pass (both operands or the product) of a transform in shared memory
template <int LG, int K, bool FWD>
__device__ __forceinline__ void fused_pass(uint32_t* buf, int gid, SharedTw tw, uint32_t p) {
    constexpr int r = prl(LG, K), R = 1 << r, LGM = lgm_of(LG, K), LGST = LGM - r, ST = 1 << LGST;
    const int j0 = gid & (ST - 1), i0 = ((gid >> LGST) << LGM) + j0;
    uint32_t x[R];
#pragma unroll
    for (int t = 0; t < R; ++t) x[t] = buf[padded_at<LGST>(i0, t)];
    if constexpr (FWD)
        dif_regs<R, ST == 1>(x, tw, j0, ST, LGM, p);
    else
        dit_regs<R, ST == 1>(x, tw, j0, ST, LGM, p);
#pragma unroll
    for (int t = 0; t < R; ++t) buf[padded_at<LGST>(i0, t)] = x[t];
}

template <int LG>
__device__ __forceinline__ void fused_body(int q, const JobDesc& J, const uint2* __restrict__ twf,
                                           const uint2* __restrict__ twi, uint32_t scw, uint32_t scws,
                                           uint32_t* err) {
    extern __shared__ __align__(16) uint8_t fu_raw[];
    FusedSmem<LG>& S = *reinterpret_cast<FusedSmem<LG>*>(fu_raw);
    constexpr int L = 1 << LG, NP = num_passes(LG), NG = L / 16;     // radix-16 groups per operand
    constexpr int T = fu_threads(LG), FU_NW = T / 32;
    static_assert(NP == 2 || NP == 3, "two or three passes");
    constexpr unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const PrimeConst pc = c_pr[q];
    const uint32_t p = pc.p;

    // twiddles of every size up to L: 16-byte asynchronous copies
    for (int i = tid; i < L; i += T) {
        const int h = i >= L / 2;
        const int e = 2 * (h ? i - L / 2 : i);
        const uint2* src = (h ? twi : twf) + (size_t)q * SBG_TW_N + e;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared((h ? S.twi : S.twf) + e));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const SharedTw sf{S.twf}, si{S.twi};
    // the reconstruction's constants, fetched while the operands are
    uint32_t touch = 0;
#pragma unroll
    for (int i = 0; i < (int)sizeof(CrtConst) / 4; i += 16) touch |= reinterpret_cast<const uint32_t*>(&c_crt)[i];
    asm volatile("" ::"r"(touch));
    pdl_enter();                               // operands and results only from here on
    // first pass: limbs -> residues -> four levels
    const int op = tid / NG, gid = tid & (NG - 1);
    const bool in_op = op < (J.sq ? 1 : 2);
    constexpr int ST0 = L / 16;
    const int xn = (int)(op ? J.bn : J.an);
    uint32_t x0[16];
    if (in_op) {
        const uint64_t* X = op ? J.b : J.a;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int n = gid + ST0 * t;
            x0[t] = n < xn ? limb_residue(__ldcg(&X[n]), pc) : 0u;
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (in_op) {
        if (xn <= L / 2)
            dif_regs<16, false, true>(x0, sf, gid, ST0, LG, p);
        else
            dif_regs<16>(x0, sf, gid, ST0, LG, p);
        uint32_t* buf = op ? S.B : S.A;
#pragma unroll
        for (int t = 0; t < 16; ++t) buf[padded_at<LG - 4>(gid, t)] = x0[t];
    }
    __syncthreads();
    if constexpr (NP == 3) {
        if (in_op) fused_pass<LG, 1, true>(op ? S.B : S.A, gid, sf, p);
        __syncthreads();
    }
    // last forward pass, product times the CRT scale, first inverse pass
    {
        constexpr int K = NP - 1, r = prl(LG, K), R = 1 << r;
        for (int g = tid; g < L / R; g += T) {
            const int i0 = g << r;
            uint32_t x[R], y[R];
#pragma unroll
            for (int t = 0; t < R; ++t) x[t] = S.A[padded_at<0>(i0, t)];
            if (J.sq) {
                dif_regs<R, true>(x, sf, 0, 1, r, p);
#pragma unroll
                for (int t = 0; t < R; ++t) y[t] = x[t];
            } else {
#pragma unroll
                for (int t = 0; t < R; ++t) y[t] = S.B[padded_at<0>(i0, t)];
                dif_regs2<R, true>(x, y, sf, 0, 1, r, p);
            }
#pragma unroll
            for (int t = 0; t < R; ++t) x[t] = mul_shoup(mont_mul(x[t], y[t], p, pc.pinv), scw, scws, p);
            dit_regs<R, true>(x, si, 0, 1, r, p);
#pragma unroll
            for (int t = 0; t < R; ++t) S.A[padded_at<0>(i0, t)] = x[t];
        }
    }
    __syncthreads();
    if constexpr (NP == 3) {
        if (tid < NG) fused_pass<LG, 1, false>(S.A, tid, si, p);
        __syncthreads();
    }
    if (tid < NG) fused_pass<LG, 0, false>(S.A, tid, si, p);
    cluster_barrier<true>();                   // every prime's residues are in shared memory

    // Coefficients -> limbs.  Limbs 0 .. nout (nout: the spill check) go to the
    // five CTAs in equal runs; a CTA's threads take two consecutive limbs each
    // from four below its run, whose coefficients the run's first limbs need.
    const int nout = (int)J.nout, off = (int)J.off, cmin = (int)J.cmin, cmax = (int)J.cmax;
    const int run = ((nout + SBG_NP) / SBG_NP + 1) & ~1;
    const int c0 = q * run, c1 = min(c0 + run, nout + 1);
    const int m0 = c0 - 4 + FU_V * tid;
    const bool on = c0 - 4 + FU_V * 32 * wid < c1;         // warps beyond the run have nothing to do
    const uint32_t inj = *(volatile uint32_t*)&g_inject;
    uint64_t lo[FU_V] = {}, mid[FU_V] = {}, z[FU_V] = {};
    uint32_t hi[FU_V] = {}, gb = 0, pb = 0, vbad = 0, wg = 0, wp = 0;
    if (on) {
        uint32_t r[FU_V][SBG_NP];
#pragma unroll
        for (int k = 0; k < SBG_NP; ++k) {
            const uint32_t base = dsmem_addr(S.A, k);
#pragma unroll
            for (int i = 0; i < FU_V; ++i) {
                const int j = m0 + i + off;
                r[i][k] = m0 + i < c1 && j >= cmin && j <= cmax ? dsmem_ld(base + 4u * pad_idx(j)) : 0u;
            }
        }
#pragma unroll
        for (int i = 0; i < FU_V; ++i) {
            const int j = m0 + i + off;
            if (inj && j >= cmin && j <= cmax &&
                (((inj & SBG_INJECT_TOP) && j == cmax) || ((inj & SBG_INJECT_MID) && j == cmin + (cmax - cmin) / 2)))
                r[i][0] ^= 1u;
            garner(r[i], lo[i], mid[i], hi[i]);
        }
        if (lane >= 30) {                      // what the warp above takes from this one
            S.xlo[wid][lane - 30] = make_ulonglong2(lo[1], mid[0]);
            S.xmid[wid][lane - 30] = mid[1];
            S.xhi[wid][lane - 30] = make_uint2(hi[0], hi[1]);
        }
    }
    __syncthreads();
    if (on) {
        uint64_t b_mid1 = __shfl_up_sync(FULL, mid[1], 1);
        uint32_t b_hi0 = __shfl_up_sync(FULL, hi[0], 1), b_hi1 = __shfl_up_sync(FULL, hi[1], 1), c_k1 = 0;
        if (lane == 0 && wid > 0) {
            uint64_t t;
            const ulonglong2 l = S.xlo[wid - 1][1];
            const uint2 h = S.xhi[wid - 1][1];
            b_mid1 = S.xmid[wid - 1][1];
            b_hi0 = h.x;
            b_hi1 = h.y;
            sum3(l.x, l.y, S.xhi[wid - 1][0].y, t, c_k1);  // the sum carry of the limb below
        }
        if (lane == 0 && wid == 0) b_mid1 = b_hi0 = b_hi1 = 0;
        uint64_t y[FU_V];
        uint32_t kk[FU_V];
        sum3(lo[0], b_mid1, b_hi0, y[0], kk[0]);
        sum3(lo[1], mid[0], b_hi1, y[1], kk[1]);
        uint32_t b_k1 = __shfl_up_sync(FULL, kk[1], 1);
        if (lane == 0) b_k1 = c_k1;
        if (m0 == 0) b_k1 = 0;                 // limb -1 carries nothing into limb 0
#pragma unroll
        for (int i = 0; i < FU_V; ++i) {
            const int m = m0 + i;
            z[i] = y[i] + (i == 0 ? b_k1 : kk[0]);
            uint32_t G = z[i] < y[i], P = z[i] == ~0ull;
            if (m >= nout) {
                if (m == nout) vbad = G | kk[i];           // must end zero with no carry beyond it
                G = 0;
                P = 0;
            }
            if (m < c0 || m >= c1) {           // not of this run: passes the carry on
                G = 0;
                P = 1;
            }
            gb |= G << i;
            pb |= P << i;
        }
        const uint32_t lG = (pb + (gb << 1)) >> FU_V, lP = pb == (1u << FU_V) - 1u;
        wg = __ballot_sync(FULL, lG & 1u);
        wp = __ballot_sync(FULL, lP);
        if (lane == 0) {
            const uint32_t G = (uint32_t)(((uint64_t)wp + (wg << 1)) >> 32) | (wg >> 31);
            S.warp[wid] = (G & 1u) | ((wp == FULL) << 1);
        }
    } else if (lane == 0) {
        S.warp[wid] = 2u;                      // identity
    }
    cluster_barrier<true>();                   // all warps' (G, P) are in shared memory
    // the carry into this warp: over the CTAs below, then this CTA's warps
    constexpr uint32_t NWM = (1u << FU_NW) - 1u;
    uint32_t v[SBG_NP], cin = 0, cw = 0;
#pragma unroll
    for (int k = 0; k < SBG_NP; ++k)
        v[k] = k <= q && lane < FU_NW ? dsmem_ld(dsmem_addr(S.warp, k) + 4 * lane) : 2u;
#pragma unroll
    for (int k = 0; k < SBG_NP; ++k) {
        const uint32_t g = __ballot_sync(FULL, v[k] & 1u) & NWM, pr = __ballot_sync(FULL, v[k] & 2u) & NWM;
        const uint32_t sum = pr + ((g << 1) | cin);
        if (k == q) cw = (sum ^ pr) >> wid;
        cin = ((sum >> (FU_NW)) | (g >> (FU_NW - 1))) & 1u;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");     // peers' memory is read
    if (on) {
        const uint32_t c = cw & 1u;
        const uint64_t sum = (uint64_t)wp + ((wg << 1) | c);
        const uint32_t cl = (((uint32_t)sum ^ wp) >> lane) & 1u;
        const uint32_t cm = (pb + ((gb << 1) | cl)) ^ pb;
#pragma unroll
        for (int i = 0; i < FU_V; ++i) {
            const int m = m0 + i;
            const uint64_t w = z[i] + ((cm >> i) & 1u);
            if (m < c0 || m >= c1) continue;
            if (m < nout)
                J.out[m] = w;
            else if (vbad | (w != 0) | (w < z[i]))
                atomicOr(err, 2u);
        }
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");       // peers may still read ours
}

template <int LG>
__global__ void __launch_bounds__(fu_threads(LG), 1) k_fused(const __grid_constant__ JobDesc J, const uint2* __restrict__ twf,
                                                   const uint2* __restrict__ twi, ScaleArg sc, uint32_t* err) {
    fused_body<LG>(blockIdx.x, J, twf, twi, sc.w[blockIdx.x], sc.ws[blockIdx.x], err);
}

// batched: one cluster per job
template <int LG>
__global__ void __launch_bounds__(fu_threads(LG), 1024 / fu_threads(LG))
    k_fused_b(const JobDesc* __restrict__ jobs, const uint2* __restrict__ twf, const uint2* __restrict__ twi, ScaleArg sc,
              uint32_t* err) {
    const int q = blockIdx.x % SBG_NP;
    fused_body<LG>(q, jobs[blockIdx.x / SBG_NP], twf, twi, sc.w[q], sc.ws[q], err);
}

// ------------------------------------------------------------------------
// Columns of 2 to 16 rows of a single product: a thread per column and prime,
// 128 threads a CTA.  The general column kernels' tiles hold 2^13 points, which
// at two rows leaves ten CTAs for both operands; here there are 320 whatever
// the length.  Launches as the profiler times them: 2 rows (8192 points) forward
// 10.6 -> 3.2 us, inverse 11.1 -> 2.9; 8 rows 6.0 -> 3.8 and 5.8 -> 3.6; 16 rows
// 5.9 -> 4.6 and 4.8 -> 5.0.  Batches keep the tiles: their jobs fill the device,
// and a CTA per 128 columns would cost them more launches than work.
// ------------------------------------------------------------------------
#define COLN_T 128
#define COLN_MAX_LG 4
#define COLN_TILES ((1 << SBG_ROW_LG) / COLN_T)
template <int LGN1>
__global__ void __launch_bounds__(COLN_T) k_coln_fwd(const uint64_t* __restrict__ a, int64_t an,
                                                     const uint64_t* __restrict__ b, int64_t bn,
                                                     const uint2* __restrict__ twf, uint32_t* __restrict__ YA,
                                                     uint32_t* __restrict__ YB) {
    constexpr int R = 1 << LGN1;
    const int tile = blockIdx.x % COLN_TILES, q = blockIdx.x / COLN_TILES % SBG_NP, op = blockIdx.x / (COLN_TILES * SBG_NP);
    const int c = tile * COLN_T + threadIdx.x;
    const PrimeConst pc = c_pr[q];
    const uint2* tw = twf + (size_t)q * SBG_TW_N;
    uint2 w[R];                                // the table's entries, read ahead of the wait
#pragma unroll
    for (int t = 0; t < R - 1; ++t) w[t] = __ldg(&tw[t]);
    pdl_enter();
    const uint64_t* X = op ? b : a;
    const int64_t xn = op ? bn : an;
    uint32_t x[R];
#pragma unroll
    for (int t = 0; t < R; ++t) x[t] = load_limb(X, xn, ((int64_t)t << SBG_ROW_LG) + c, pc);
    dif_regs<R, true>(x, SharedTw{w}, 0, 1, LGN1, pc.p);
    uint32_t* Y = (op ? YB : YA) + ((size_t)q << (LGN1 + SBG_ROW_LG)) + c;
#pragma unroll
    for (int t = 0; t < R; ++t) Y[t << SBG_ROW_LG] = x[t];
}

template <int LGN1>
__global__ void __launch_bounds__(COLN_T) k_coln_inv(uint32_t* __restrict__ YA, const uint2* __restrict__ twi) {
    constexpr int R = 1 << LGN1;
    const int tile = blockIdx.x % COLN_TILES, q = blockIdx.x / COLN_TILES;
    const PrimeConst pc = c_pr[q];
    const uint2* tw = twi + (size_t)q * SBG_TW_N;
    uint2 w[R];
#pragma unroll
    for (int t = 0; t < R - 1; ++t) w[t] = __ldg(&tw[t]);
    pdl_enter();
    uint32_t* Y = YA + ((size_t)q << (LGN1 + SBG_ROW_LG)) + tile * COLN_T + threadIdx.x;
    uint32_t x[R];
#pragma unroll
    for (int t = 0; t < R; ++t) x[t] = __ldcg(&Y[t << SBG_ROW_LG]);
    dit_regs<R, true>(x, SharedTw{w}, 0, 1, LGN1, pc.p);
#pragma unroll
    for (int t = 0; t < R; ++t) Y[t << SBG_ROW_LG] = x[t];
}
#define SBG_COLN_CASES(X) X(1) X(2) X(3) X(4)

// ------------------------------------------------------------------------
// Columns of 3 * 2^m rows, m = 0 .. 3 (transforms of 3 * 2^12 .. 3 * 2^15
// points): a thread per column holds all its rows; the radix-3 level over the
// thirds, then a 2^m-point DIF per third, as in the longer 3 * 2^m columns.
// CPT columns per thread: one for a lone product, more for a batch's jobs.
// ------------------------------------------------------------------------
#define COL3N_MAX 3
__host__ __device__ constexpr int col3n_cpt(int m) { return m <= 1 ? 4 : (m == 2 ? 2 : 1); }
__host__ __device__ constexpr int col3n_tiles(int cpt) { return COLN_TILES / cpt; }
template <int M3, int CPT>
__device__ __forceinline__ void col3n_fwd_body(int q, int tile, const uint64_t* __restrict__ X, int64_t xn,
                                               const uint2* __restrict__ twf, const Radix3Arg& r3,
                                               uint32_t* __restrict__ Y) {
    constexpr int M = 1 << M3;
    const PrimeConst pc = c_pr[q];
    const uint2* tw = twf + (size_t)q * SBG_TW_N;
    const uint2* t3 = r3.t3 + ((size_t)q << (M3 + 1));
    Y += (size_t)q * (3 * M) << SBG_ROW_LG;
#pragma unroll 1
    for (int i = 0; i < CPT; ++i) {
        const int c = (tile * CPT + i) * COLN_T + threadIdx.x;
        uint32_t x[M], y[M], z[M];
#pragma unroll
        for (int r = 0; r < M; ++r) {
            x[r] = load_limb(X, xn, ((int64_t)r << SBG_ROW_LG) + c, pc);
            y[r] = load_limb(X, xn, ((int64_t)(r + M) << SBG_ROW_LG) + c, pc);
            z[r] = load_limb(X, xn, ((int64_t)(r + 2 * M) << SBG_ROW_LG) + c, pc);
        }
#pragma unroll
        for (int r = 0; r < M; ++r)
            r3_dif(x[r], y[r], z[r], r3.w[q], r3.ws[q], __ldg(&t3[r]), __ldg(&t3[2 * r]), pc.p);
        if constexpr (M > 1) {
            dif_regs2<M, true>(x, y, tw, 0, 1, M3, pc.p);
            dif_regs<M, true>(z, tw, 0, 1, M3, pc.p);
        }
        uint32_t* out = Y + c;
#pragma unroll
        for (int r = 0; r < M; ++r) {
            out[r << SBG_ROW_LG] = x[r];
            out[(r + M) << SBG_ROW_LG] = y[r];
            out[(r + 2 * M) << SBG_ROW_LG] = z[r];
        }
    }
}
template <int M3, int CPT>
__device__ __forceinline__ void col3n_inv_body(int q, int tile, uint32_t* __restrict__ Y, const uint2* __restrict__ twi,
                                               const Radix3Arg& r3) {
    constexpr int M = 1 << M3;
    const PrimeConst pc = c_pr[q];
    const uint2* tw = twi + (size_t)q * SBG_TW_N;
    const uint2* t3 = r3.t3 + ((size_t)q << (M3 + 1));
    Y += (size_t)q * (3 * M) << SBG_ROW_LG;
#pragma unroll 1
    for (int i = 0; i < CPT; ++i) {
        uint32_t* col = Y + (tile * CPT + i) * COLN_T + threadIdx.x;
        uint32_t x[M], y[M], z[M];
#pragma unroll
        for (int r = 0; r < M; ++r) {
            x[r] = __ldcg(&col[r << SBG_ROW_LG]);
            y[r] = __ldcg(&col[(r + M) << SBG_ROW_LG]);
            z[r] = __ldcg(&col[(r + 2 * M) << SBG_ROW_LG]);
        }
        if constexpr (M > 1) {
            dit_regs2<M, true>(x, y, tw, 0, 1, M3, pc.p);
            dit_regs<M, true>(z, tw, 0, 1, M3, pc.p);
        }
#pragma unroll
        for (int r = 0; r < M; ++r) {
            r3_dit(x[r], y[r], z[r], r3.w[q], r3.ws[q], __ldg(&t3[r]), __ldg(&t3[2 * r]), pc.p);
            col[r << SBG_ROW_LG] = x[r];
            col[(r + M) << SBG_ROW_LG] = y[r];
            col[(r + 2 * M) << SBG_ROW_LG] = z[r];
        }
    }
}
template <int M3>
__global__ void __launch_bounds__(COLN_T) k_col3n_fwd(const uint64_t* __restrict__ a, int64_t an,
                                                      const uint64_t* __restrict__ b, int64_t bn,
                                                      const uint2* __restrict__ twf, Radix3Arg r3,
                                                      uint32_t* __restrict__ YA, uint32_t* __restrict__ YB) {
    pdl_enter();
    const int tile = blockIdx.x % COLN_TILES, q = blockIdx.x / COLN_TILES % SBG_NP, op = blockIdx.x / (COLN_TILES * SBG_NP);
    col3n_fwd_body<M3, 1>(q, tile, op ? b : a, op ? bn : an, twf, r3, op ? YB : YA);
}
template <int M3>
__global__ void __launch_bounds__(COLN_T) k_col3n_inv(uint32_t* __restrict__ YA, const uint2* __restrict__ twi,
                                                      Radix3Arg r3) {
    pdl_enter();
    col3n_inv_body<M3, 1>(blockIdx.x / COLN_TILES, blockIdx.x % COLN_TILES, YA, twi, r3);
}
// batched: blocks (job, operand, prime, tile), job slowest
template <int M3>
__global__ void __launch_bounds__(COLN_T) k_col3n_fwd_b(const JobDesc* __restrict__ jobs, const uint2* __restrict__ twf,
                                                        Radix3Arg r3) {
    pdl_enter();
    constexpr int CPT = col3n_cpt(M3), NT = col3n_tiles(CPT), PER_JOB = 2 * SBG_NP * NT;
    const JobDesc& J = jobs[blockIdx.x / PER_JOB];
    const int r = blockIdx.x % PER_JOB, op = r / (SBG_NP * NT);
    if (op && J.sq) return;
    uint32_t* Y = J.ws + (op ? (size_t)SBG_NP * (3 << M3) << SBG_ROW_LG : 0);
    col3n_fwd_body<M3, CPT>(r / NT % SBG_NP, r % NT, op ? J.b : J.a, op ? J.bn : J.an, twf, r3, Y);
}
template <int M3>
__global__ void __launch_bounds__(COLN_T) k_col3n_inv_b(const JobDesc* __restrict__ jobs, const uint2* __restrict__ twi,
                                                        Radix3Arg r3) {
    pdl_enter();
    constexpr int CPT = col3n_cpt(M3), NT = col3n_tiles(CPT), PER_JOB = SBG_NP * NT;
    const int r = blockIdx.x % PER_JOB;
    col3n_inv_body<M3, CPT>(r / NT, r % NT, jobs[blockIdx.x / PER_JOB].ws, twi, r3);
}
#define SBG_COL3N_CASES(X) X(0) X(1) X(2) X(3)

#define SBG_FUSED_CASES(X) X(8) X(9) X(10) X(11) X(12)

// ------------------------------------------------------------------------
// The row kernel of few rows.  k_row12 runs both operands of a row on 256
// threads, four CTAs per SM, its twiddles read through L1: the right form when
// rows queue for the SMs, but a lone row takes it 28,000 clocks, most of them
// spent waiting for twiddles that no other CTA has brought to L1.  Here a row
// has 512 threads, an operand to each half, and its twiddles staged in shared
// memory -- before the previous kernel of the chain is waited for, as the
// tables are older than that.  Device time a launch, 10 to 80 rows: 14.5 -> 9.9 us.
// Beyond one row per SM k_row12 wins (160 rows: 17.3 us here, 15 to 17 there).
// ------------------------------------------------------------------------
#define ROWL_MAX 148
struct RowlSmem {
    uint32_t A[padded_len(ROW_N)];
    uint32_t B[padded_len(ROW_N)];
    uint2 twf[ROW_N];
    uint2 twi[ROW_N];
    uint2 f[16];                               // four-step twiddle steps, w_L^(256 k1 t)
    uint2 i[16];                               // their inverses times the CRT scale
};

// more than half an SM's shared memory: while the column kernel's CTAs are
// still leaving, the scheduler would put two rows on one SM and none on another
// (40 rows: 13 instead of 9 us)
#define ROWL_SMEM (size_t)(120 << 10)
static_assert(sizeof(RowlSmem) <= ROWL_SMEM, "row tables");

template <bool BATCH>
__global__ void __launch_bounds__(FU_T, 1) k_rowl(uint32_t* __restrict__ YA, const uint32_t* __restrict__ YB, int sq,
                                                  const JobDesc* __restrict__ jobs, int lgN1, int m3, FsTables fsf,
                                                  FsTables fsi, ScaleArg sc, const uint2* __restrict__ twf,
                                                  const uint2* __restrict__ twi, uint32_t* flags, int64_t nflags) {
    extern __shared__ __align__(16) uint8_t fu_raw[];
    RowlSmem& S = *reinterpret_cast<RowlSmem*>(fu_raw);
    constexpr int LG = ROW_LG;
    const int n1 = m3 >= 0 ? 3 << m3 : 1 << lgN1;
    const int per_job = SBG_NP * n1;
    const int r = BATCH ? blockIdx.x % per_job : blockIdx.x;
    const int q = r / n1, row = r - q * n1;
    const int tid = threadIdx.x, op = tid >> 8, gid = tid & 255;
    const PrimeConst pc = c_pr[q];
    const uint32_t p = pc.p;
    for (int k = tid; k < ROW_N; k += FU_T) {
        const int h = k >= ROW_N / 2;
        const int e = 2 * (h ? k - ROW_N / 2 : k);
        const uint2* src = (h ? twi : twf) + (size_t)q * SBG_TW_N + e;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared((h ? S.twi : S.twf) + e));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const SharedTw sf{S.twf}, si{S.twi};
    // four-step twiddles of this row, as in row_body
    const uint32_t k1 = m3 >= 0 ? 3u * bitrev((uint32_t)row & ((1u << m3) - 1u), m3) + ((uint32_t)row >> m3)
                                : bitrev((uint32_t)row, lgN1);
    if (tid < 32) {
        const uint32_t e = k1 * 256u * (uint32_t)(tid & 15);
        const uint32_t v = tid < 16 ? fs_value(fsf, q, e, p) : mul_shoup(fs_value(fsi, q, e, p), sc.w[q], sc.ws[q], p);
        (tid < 16 ? S.f : S.i)[tid & 15] = make_uint2(v, shoup_fast(v, pc));
    }
    const uint32_t eb = k1 * (uint32_t)gid;
    const uint32_t bf = fs_value(fsf, q, eb, p), bfs = shoup_fast(bf, pc);
    const uint32_t bi = fs_value(fsi, q, eb, p), bis = shoup_fast(bi, pc);
    pdl_enter();
    clear_flags(flags, nflags);
    if (BATCH) {
        const JobDesc& J = jobs[blockIdx.x / per_job];
        YA = J.ws;
        YB = J.ws + (size_t)SBG_NP * n1 * ROW_N;
        sq = J.sq;
    }
    const size_t base = ((size_t)q * n1 + row) * ROW_N;
    const bool on = op == 0 || !sq;
    uint32_t x[16];
    if (on) {
        const uint32_t* src = (op ? YB : YA) + base + gid;
#pragma unroll
        for (int t = 0; t < 16; ++t) x[t] = __ldcg(src + 256 * t);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    uint32_t* buf = op ? S.B : S.A;
    if (on) {
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const uint2 s = S.f[t];
            x[t] = mul_shoup(mul_shoup(x[t], s.x, s.y, p), bf, bfs, p);
        }
        dif_regs<16>(x, sf, gid, 256, LG, p);
#pragma unroll
        for (int t = 0; t < 16; ++t) buf[padded_at<8>(gid, t)] = x[t];
    }
    __syncthreads();
    if (on) fused_pass<LG, 1, true>(buf, gid, sf, p);
    __syncthreads();
    if (op == 0) {
        // last forward pass, product, first inverse pass
        const int i0 = gid << 4;
        uint32_t y[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) x[t] = S.A[padded_at<0>(i0, t)];
        if (sq) {
            dif_regs<16, true>(x, sf, 0, 1, 4, p);
#pragma unroll
            for (int t = 0; t < 16; ++t) x[t] = mont_mul(x[t], x[t], p, pc.pinv);
        } else {
#pragma unroll
            for (int t = 0; t < 16; ++t) y[t] = S.B[padded_at<0>(i0, t)];
            dif_regs2<16, true>(x, y, sf, 0, 1, 4, p);
#pragma unroll
            for (int t = 0; t < 16; ++t) x[t] = mont_mul(x[t], y[t], p, pc.pinv);
        }
        dit_regs<16, true>(x, si, 0, 1, 4, p);
#pragma unroll
        for (int t = 0; t < 16; ++t) S.A[padded_at<0>(i0, t)] = x[t];
    }
    __syncthreads();
    if (op == 0) fused_pass<LG, 1, false>(S.A, gid, si, p);
    __syncthreads();
    if (op == 0) {
#pragma unroll
        for (int t = 0; t < 16; ++t) x[t] = S.A[padded_at<8>(gid, t)];
        dit_regs<16>(x, si, gid, 256, LG, p);
        uint32_t* dst = YA + base + gid;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const uint2 s = S.i[t];
            dst[256 * t] = mul_shoup(mul_shoup(x[t], s.x, s.y, p), bi, bis, p);
        }
    }
}

static cudaError_t fused_attr() {
    cudaError_t e = cudaSuccess;
#define SBG_FUSED_ATTR(n) \
    if (e == cudaSuccess) \
        e = cudaFuncSetAttribute(k_fused<n>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FusedSmem<n>)); \
    if (e == cudaSuccess) \
        e = cudaFuncSetAttribute(k_fused_b<n>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FusedSmem<n>));
    SBG_FUSED_CASES(SBG_FUSED_ATTR)
#undef SBG_FUSED_ATTR
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rowl<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ROWL_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rowl<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ROWL_SMEM);
    return e;
}

}  // namespace sbg
