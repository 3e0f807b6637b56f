// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) in float32 on the fifth-generation tensor cores: the matrix product of the 32-bit path.
//
// A 32-bit number of 2^-109 or more is the sum of three bfloat16 ones, exactly: its value rounded to 8 bits, what is left rounded
// to 8 bits, and the rest (24 bits in all; Dekker's splitting, with three parts).  Of the nine products of two such numbers the six that
// matter are formed by tcgen05.mma (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi; the others are 2^-24 of the result and
// below), each exact before it is added, the small ones first.  The tensor core cuts off what does not fit into an accumulator where
// a multiply-add rounds, so an accumulator takes 32 k only and is then added, rounded, to a sum in a register.  Error against 64
// bits (2-norm, normal operands), multiply-adds one after another in parts (gemm_f32.cu) and this: K = 1024 2.1e-7 and 8.9e-8, 3072 2.6e-7
// and 1.05e-7, 9728 4.5e-7 and 1.4e-7.
//
// Order of a sum: k is cut into at most eight parts of equal length, by K alone (gt_parts); within a part runs of 32 k are added
// in ascending order, then the parts' sums.  Every tile and split below keeps that order, so a row's result does not
// depend on how many rows the call has.
//
// A block forms a tile of 128 rows of W (the M side of the product: out^T = W A^T) by up to 128 rows of A.  Its 512 threads
// fetch 64 k of both as float32 (16 bytes a load, ahead of their use), split them and store the three parts into shared memory in the
// layout that the tensor core reads (128-byte swizzle); one elected lane issues the products; while they run all threads add the
// accumulators of the chunk before and split the next one.  Two stages, two sets of accumulators.  Few tiles: the parts of k go
// to the blocks of a cluster, one, two or four to a block, which add them through distributed shared memory.
//
// What bounds it: up to some 64 rows the traffic in shared memory (1.2 us a chunk: six reads of W's tile by the tensor core, the
// splitting's stores, the copies), above that the splitting and the products about alike.  (With 256 threads two warps a scheduler waited on each
// other: 40 % of the issue slots used, 1.4 to 2.9 us a chunk.)  Measurements: at vx_gemm_f32_takes_tc below.
//
// What three parts cannot hold is formed again by multiply-adds in ascending k: sums that are no ordinary numbers (an infinity or
// NaN among the operands, a sum that overflows), so that infinities and NaN come out as they do there; and those to which what
// bfloat16 loses below 2^-126 may matter.  An operand loses less than 2^-125, so a sum of K products loses less than
// K 2^-94 while all operands are below 2^30: nothing, to a sum of 2^-50 or more (K up to 2^20).  Hence: sums below 2^-50 (0 included, unless
// a row is all zeros) and sums with an operand of 2^30 or more.  Both follow from the sum's own two rows.  (Rows are only searched where a
// tile holds so large an operand: a maximum in the loop, 0 to 3 %; 300 x 6144 x 1024 40.9 us without it, 41.7, as sums of squares 46.2.)
#include <cooperative_groups.h>

#include "gemm_f32.cuh"
#include "tcgen05_gemm.cuh"

namespace cg = cooperative_groups;

#define GT_BN 128      // rows of W a tile takes
#define GT_BK 64       // k of a chunk
#define GT_RUN 32      // k of an accumulator
#define GT_THREADS 512
#define GT_STEP 32     // rows that the block's warps fetch side by side (two a warp)
#define GT_MAX_PARTS 8
#define GT_W_BYTES (GT_BN * GT_BK * 2)

// The three bfloat16 parts of two neighbouring numbers, packed.
__device__ __forceinline__ void gt_split2(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    hi = reinterpret_cast<const unsigned&>(h);
    const float x1 = x - __uint_as_float(hi << 16), y1 = y - __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 m = __floats2bfloat162_rn(x1, y1);
    mid = reinterpret_cast<const unsigned&>(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x1 - __uint_as_float(mid << 16), y1 - __uint_as_float(mid & 0xffff0000u));
    lo = reinterpret_cast<const unsigned&>(l);
}

// Four k of a row, zeros beyond the `left` that there are.
template <bool VEC>
__device__ __forceinline__ float4 gt_fetch(const float* __restrict__ at, int left, bool in) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!in || left <= 0) return v;
    if (VEC && left >= 4) return *reinterpret_cast<const float4*>(at);
    v.x = at[0];
    if (left > 1) v.y = at[1];
    if (left > 2) v.z = at[2];
    if (left > 3) v.w = at[3];
    return v;
}

// Four k to their places in the swizzled layout: `at` and, `part_bytes` apart, the other two parts.
__device__ __forceinline__ void gt_store(unsigned char* at, unsigned part_bytes, const float4& v) {
    uint2 h, m, l;
    gt_split2(v.x, v.y, h.x, m.x, l.x);
    gt_split2(v.z, v.w, h.y, m.y, l.y);
    *reinterpret_cast<uint2*>(at) = h;
    *reinterpret_cast<uint2*>(at + part_bytes) = m;
    *reinterpret_cast<uint2*>(at + 2 * part_bytes) = l;
}

// `left` k of a row (four at most) on their way into the thread's own place in shared memory, zeros for the rest.
template <bool VEC>
__device__ __forceinline__ void gt_copy(unsigned dst, const float* __restrict__ at, int left) {
    if (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(at), "r"(max(0, min(4, left)) * 4) : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst + 4 * e), "l"(e < left ? at + e : at), "r"(e < left ? 4 : 0) : "memory");
    }
}

// N columns of 32 lanes of tensor memory (the caller waits).
template <int N>
__device__ __forceinline__ void gt_ld(unsigned taddr, unsigned* r) {
    if (N == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
    else if (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr) : "memory");
}

struct GtCall {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc, batch;
    long long sa, sw, sc;
    int w_ready;
    int* error;
};

// The larger of `top` and four numbers' magnitudes (a NaN is passed over).
__device__ __forceinline__ float gt_top(float top, const float4& v) {
    asm("{\n .reg .f32 a, b;\n abs.f32 a, %1;\n abs.f32 b, %2;\n max.f32 %0, %0, a, b;\n abs.f32 a, %3;\n abs.f32 b, %4;\n max.f32 %0, %0, a, b;\n}\n"
        : "+f"(top) : "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
    return top;
}
__device__ __forceinline__ bool gt_any(const float* a, int K, float least) {   // (whether a magnitude is `least` or more)
    for (int k = 0; k < K; ++k)
        if (fabsf(a[k]) >= least) return true;
    return false;
}
// The tensor cores' sum `v` of two rows if they could form it, else the sum by multiply-adds one after another.  `huge`: an operand
// of GT_HUGE or more is somewhere in the tile.
#define GT_HUGE 1.073741824e9f   // 2^30
#define GT_TINY 8.8817842e-16f   // 2^-50
__device__ __noinline__ float gt_careful(const float* a, const float* b, int K, float v, bool huge) {
    const float size = fabsf(v);
    bool again = !(size < INFINITY);
    if (!again && size < GT_TINY) again = size > 0.f || (gt_any(a, K, 1.4e-45f) && gt_any(b, K, 1.4e-45f));
    if (!again && huge) again = gt_any(a, K, GT_HUGE) || gt_any(b, K, GT_HUGE);
    if (!again) return v;
    v = 0.f;
#pragma unroll 8
    for (int k = 0; k < K; ++k) v = fmaf(a[k], b[k], v);
    return v;
}

__host__ __device__ constexpr int gt_ahead(int bm) { return bm <= 32 ? 2 : (bm <= 64 ? 1 : 0); }
__host__ __device__ constexpr int gt_xsteps(int bm) { return (bm + GT_STEP - 1) / GT_STEP; }
__host__ __device__ constexpr int gt_stages_bytes(int bm) { return 2 * (3 * GT_W_BYTES + 3 * bm * 128); }
__host__ __device__ constexpr int gt_smem(int bm) {
    return gt_stages_bytes(bm) + gt_ahead(bm) * (GT_BN / GT_STEP + gt_xsteps(bm)) * GT_THREADS * 16;
}

// BM: rows of A a tile has room for; `bm` of them (a multiple of 16) are used.  PER: parts of k that a block of the cluster sums up,
// each by itself (0: no cluster, the block adds all parts).
template <int BM, bool VEC, int PER>
__global__ void __launch_bounds__(GT_THREADS, 1)
gemm_f32_tc_kernel(GtCall g, int bm, int parts, int part_len) {
    constexpr bool SPLIT = PER > 0;
    constexpr int STAGE = 3 * GT_W_BYTES + 3 * BM * 128, AHEAD = gt_ahead(BM);
    constexpr int COLS = BM / 4, LDN = COLS < 16 ? COLS : 16;      // columns of a warp, of a load from tensor memory
    constexpr int RUNS = GT_BK / GT_RUN, TMEM = 2 * RUNS * BM;
    constexpr int WSTEPS = GT_BN / GT_STEP, XSTEPS = gt_xsteps(BM);
    extern __shared__ unsigned char gt_raw[];
    __shared__ __align__(8) unsigned long long done[2];
    __shared__ unsigned tmem_s;
    __shared__ int failed, huge_s;
    unsigned char* tiles = (unsigned char*)(((uintptr_t)gt_raw + 1023) & ~(uintptr_t)1023);
    const float* A = g.A + (size_t)blockIdx.z * g.sa;
    const float* W = g.W + (size_t)blockIdx.z * g.sw;
    float* C = g.C + (size_t)blockIdx.z * g.sc;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int blocks = SPLIT ? (parts + PER - 1) / (SPLIT ? PER : 1) : 1;   // of the cluster
    const int rank = SPLIT ? (int)blockIdx.x % blocks : 0;
    const int n0 = (SPLIT ? (int)blockIdx.x / blocks : (int)blockIdx.x) * GT_BN, m0 = blockIdx.y * bm;
    const int kbeg = SPLIT ? rank * PER * part_len : 0, kend = SPLIT ? min(g.K, kbeg + PER * part_len) : g.K;
    const int chunks = (kend - kbeg + GT_BK - 1) / GT_BK;
    // a warp's 32 lanes fetch 64 k of two rows at a time: row GT_STEP i + fr, columns 4 c4
    const int fr = warp * 2 + (lane >> 4), c4 = lane & 15;

    if (threadIdx.x == 0) {
        tc_mbar_init(tc_smem_u32(&done[0]), 1);
        tc_mbar_init(tc_smem_u32(&done[1]), 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // What a thread will split it fetches itself: AHEAD chunks on their way into places of its own in shared memory, or (where
    // those do not fit) one in registers.  Rows beyond the matrices are taken as zeros.
    float4 w[WSTEPS], x[XSTEPS];
    unsigned char* const own = tiles + 2 * STAGE + threadIdx.x * 16;
    const unsigned own_addr = tc_smem_u32(own);
    constexpr unsigned STEP = GT_THREADS * 16, SLOT = (WSTEPS + XSTEPS) * STEP;
    const float *wrow[WSTEPS], *xrow[XSTEPS];
    unsigned there = 0;   // bit i: W's row of step i, bit 16 + i: A's
#pragma unroll
    for (int i = 0; i < WSTEPS; ++i) {
        const int n = n0 + GT_STEP * i + fr;
        there |= n < g.N ? 1u << i : 0u;
        wrow[i] = W + (size_t)(n < g.N ? n : 0) * g.ldw + kbeg + 4 * c4;
    }
#pragma unroll
    for (int i = 0; i < XSTEPS; ++i) {
        const int r = GT_STEP * i + fr, m = m0 + r;
        const bool in = r < bm && m < g.M;
        there |= in ? 1u << (16 + i) : 0u;
        xrow[i] = A + (size_t)(in ? m : 0) * g.lda + kbeg + 4 * c4;
    }
    const int left0 = kend - kbeg - 4 * c4;   // k that are left from the thread's first on
    auto fetch_w = [&](int c) {
        const int left = left0 - c * GT_BK;
        const unsigned slot = own_addr + (AHEAD ? c % (AHEAD ? AHEAD : 1) : 0) * SLOT;
#pragma unroll
        for (int i = 0; i < WSTEPS; ++i) {
            const bool in = there >> i & 1;
            const float* at = wrow[i] + (left > 0 ? c * GT_BK : -4 * c4);   // (nothing left: an address inside the row all the same)
            if (AHEAD) gt_copy<VEC>(slot + i * STEP, at, in ? left : 0);
            else w[i] = gt_fetch<VEC>(at, left, in);
        }
    };
    auto fetch_x = [&](int c) {
        const int left = left0 - c * GT_BK;
        const unsigned slot = own_addr + (AHEAD ? c % (AHEAD ? AHEAD : 1) : 0) * SLOT;
#pragma unroll
        for (int i = 0; i < XSTEPS; ++i) {
            const bool in = there >> (16 + i) & 1;
            const float* at = xrow[i] + (left > 0 ? c * GT_BK : -4 * c4);
            if (AHEAD) gt_copy<VEC>(slot + (WSTEPS + i) * STEP, at, in ? left : 0);
            else x[i] = gt_fetch<VEC>(at, left, in);
        }
    };
    // a W that the caller calls ready depends on no earlier kernel: its first chunks are asked for before the wait
    if (!g.w_ready) pdl_wait();
#pragma unroll
    for (int c = 0; c < (AHEAD ? AHEAD : 1); ++c)
        if (c < chunks) fetch_w(c);
    pdl_wait();   // (a second time it returns at once)
#pragma unroll
    for (int c = 0; c < (AHEAD ? AHEAD : 1); ++c) {
        if (c < chunks) fetch_x(c);
        if (AHEAD) asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    if (warp == 0) {   // (after the wait: the kernel before may hold tensor memory)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_s)), "r"((unsigned)TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdl_trigger();
    const unsigned tmem = tmem_s;

    constexpr int KEPT = SPLIT ? PER - 1 : 1;   // the sum of the parts so far; in a cluster each part before the block's last
    float acc[COLS], total[KEPT ? KEPT : 1][KEPT ? COLS : 1];
    float top = 0.f;
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
#pragma unroll
    for (int p = 0; p < KEPT; ++p)
#pragma unroll
        for (int j = 0; j < COLS; ++j) total[p][j] = 0.f;
    const int col0 = (warp >> 2) * COLS;   // this warp's columns (rows of A), its lanes (rows of W) are 32 (warp % 4) ..
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(bm >> 3) << 17) | ((unsigned)(GT_BN >> 4) << 24);
    int left = part_len / GT_BK, kept = 0;   // chunks until the part ends; parts that have
    bool ok = true;
    // adds chunk c's accumulators
    auto drain = [&](int c) {
        ok = ok && tc_warp_wait(tc_smem_u32(&done[c & 1]), (unsigned)((c >> 1) & 1));   // (once one has run out no further one is waited for)
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (col0 < bm) {   // (uniform)
#pragma unroll
            for (int run = 0; run < RUNS; ++run) {
                const unsigned at = tmem + (unsigned)(((c & 1) * RUNS + run) * BM + col0) + ((unsigned)((warp & 3) * 32) << 16);
#pragma unroll
                for (int j = 0; j < COLS; j += LDN) {
                    unsigned r[LDN];
                    gt_ld<LDN>(at + j, r);   // (columns past bm are not stored)
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int i = 0; i < LDN; ++i) acc[j + i] += __uint_as_float(r[i]);
                }
            }
        }
        if (KEPT && (--left == 0 || c + 1 == chunks) && !(SPLIT && c + 1 == chunks)) {   // (a cluster's block keeps its last part in acc)
            left = part_len / GT_BK;
#pragma unroll
            for (int p = 0; p < KEPT; ++p)
                if (!SPLIT || p == kept) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j) total[p][j] += acc[j];
                }
            ++kept;
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    };
    const unsigned place = (unsigned)(fr * 128 + (((c4 >> 1) ^ (fr & 7)) << 4) + (c4 & 1) * 8);   // in a part of a stage (GT_STEP rows on: 4 KB on)
    for (int c = 0; c < chunks; ++c) {
        // (the stage is free: chunk c - 2, which had it, was drained after its products had ended)
        unsigned char* st = tiles + (c & 1) * STAGE;
        unsigned char* sx = st + 3 * GT_W_BYTES;
        if (AHEAD) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD ? AHEAD - 1 : 0) : "memory");
            const unsigned char* slot = own + (c % (AHEAD ? AHEAD : 1)) * SLOT;
#pragma unroll
            for (int i = 0; i < WSTEPS; ++i) w[i] = *reinterpret_cast<const float4*>(slot + i * STEP);
#pragma unroll
            for (int i = 0; i < XSTEPS; ++i) x[i] = *reinterpret_cast<const float4*>(slot + (WSTEPS + i) * STEP);
        }
#pragma unroll
        for (int i = 0; i < WSTEPS; ++i) {
            top = gt_top(top, w[i]);
            gt_store(st + place + i * GT_STEP * 128, GT_W_BYTES, w[i]);
        }
#pragma unroll
        for (int i = 0; i < XSTEPS; ++i) {
            top = gt_top(top, x[i]);
            if (GT_STEP * i + fr < bm) gt_store(sx + place + i * GT_STEP * 128, BM * 128, x[i]);
        }
        if (c + (AHEAD ? AHEAD : 1) < chunks) {
            fetch_w(c + (AHEAD ? AHEAD : 1));
            fetch_x(c + (AHEAD ? AHEAD : 1));
        }
        if (AHEAD) asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned wa = tc_desc_lo(tc_smem_u32(st)), xa = tc_desc_lo(tc_smem_u32(sx)), d0 = tmem + (unsigned)((c & 1) * RUNS * BM);
            if (tc_elect()) {
#pragma unroll
                for (int run = 0; run < RUNS; ++run) {
                    const unsigned d = d0 + (unsigned)(run * BM), wr = wa + (run * GT_RUN * 2 >> 4), xr = xa + (run * GT_RUN * 2 >> 4);
                    constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, XP[6] = {0, 2, 1, 0, 1, 0};   // parts of W and of A: hi, mid, lo
#pragma unroll
                    for (int p = 0; p < 6; ++p)
                        tc_mma_run<1, GT_RUN / 16>(d, wr + (WP[p] * GT_W_BYTES >> 4), xr + (XP[p] * BM * 128 >> 4), idesc, p > 0);
                }
                tc_commit(tc_smem_u32(&done[c & 1]));
            }
            __syncwarp();
        }
        if (c) drain(c - 1);
    }
    drain(chunks - 1);
    if (AHEAD) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (!ok && lane == 0) {
        failed = 1;
        if (g.error) atomicExch(g.error, TC_ERR_EPILOGUE);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    bool huge = __syncthreads_or(top >= GT_HUGE);   // (everyone has read the tensor memory, and the tensor core the stages)
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((unsigned)TMEM) : "memory");
    }
    const bool bad = failed != 0;   // (a wait ran out: NaN)
    // the sum of row m of A and row n of W as it is written
    auto finish = [&](float v, int m, int n) {
        const float size = fabsf(v);
        if (bad) v = __int_as_float(0x7fc00000);
        else if (huge || !(size < INFINITY && size >= GT_TINY)) v = gt_careful(A + (size_t)m * g.lda, W + (size_t)n * g.ldw, g.K, v, huge);
        C[(size_t)m * g.ldc + n] = v + (g.bias ? g.bias[n] : 0.f);
    };
    const int row = (warp & 3) * 32 + lane;
    if (!SPLIT) {
        if (n0 + row < g.N) {
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                if (col0 + j < bm && m0 + col0 + j < g.M) finish(total[0][KEPT ? j : 0], m0 + col0 + j, n0 + row);
        }
        return;
    }
    float* sums = reinterpret_cast<float*>(tiles);   // [part][bm][128]: this block's parts' sums, in place of the stages
#pragma unroll
    for (int p = 0; p < (SPLIT ? PER : 1); ++p)
        if (p <= kept) {
#pragma unroll
            for (int j = 0; j < COLS; ++j)
                if (col0 + j < bm) sums[(p * bm + col0 + j) * GT_BN + row] = bad ? __int_as_float(0x7fc00000) : (p == kept || !KEPT ? acc[j] : total[p < KEPT ? p : 0][KEPT ? j : 0]);
        }
    if (threadIdx.x == 0) huge_s = huge;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int p = 0; p < blocks; ++p) huge = huge || *cluster.map_shared_rank(&huge_s, p);
    const int used = min(bm, g.M - m0) * GT_BN;
    for (int e = rank * GT_THREADS + threadIdx.x; e < used; e += blocks * GT_THREADS) {
        const int n = n0 + e % GT_BN;
        if (n >= g.N) continue;
        float v = 0.f;
        for (int p = 0; p < parts; ++p) v += cluster.map_shared_rank(sums, p / (SPLIT ? PER : 1))[p % (SPLIT ? PER : 1) * bm * GT_BN + e];
        finish(v, m0 + e / GT_BN, n);
    }
    cluster.sync();   // (a block's sums are read until here)
}

// k's parts and their length (a multiple of 64): of 256 k at least, eight parts at most.  No part is empty.
static void gt_parts(int K, int* parts, int* len) {
    int p = K / 256;
    p = p < 1 ? 1 : (p > GT_MAX_PARTS ? GT_MAX_PARTS : p);
    *len = ((K + p - 1) / p + GT_BK - 1) / GT_BK * GT_BK;
    *parts = (K + *len - 1) / *len;
}

// `blocks`: of a cluster (1: none).
template <int BM>
static cudaLaunchConfig_t gt_config(const GtCall& g, int bm, int blocks, cudaLaunchAttribute (&attr)[2], cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.N + GT_BN - 1) / GT_BN * blocks), (unsigned)((g.M + bm - 1) / bm), (unsigned)g.batch);
    cfg.blockDim = dim3(GT_THREADS);
    cfg.dynamicSmemBytes = gt_smem(BM) + 1024;
    cfg.stream = stream;
    int n = 0;
    if (blocks > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = blocks;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (vx_pdl_is_enabled() && ((vx_pdl_mask() >> VX_K_GEMM) & 1)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cfg;
}

template <int BM, bool VEC, int PER>
static int gt_launch(const GtCall& g, int bm, int parts, int len, cudaStream_t stream) {
    auto kernel = gemm_f32_tc_kernel<BM, VEC, PER>;
    static_assert(gt_stages_bytes(BM) >= PER * BM * GT_BN * 4, "the parts' sums fit into the stages");
    static bool configured[VX_MAX_DEVICES];
    if (int rc = vx_configure_smem(kernel, gt_smem(BM) + 1024, configured)) return rc;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = gt_config<BM>(g, bm, PER ? (parts + PER - 1) / (PER ? PER : 1) : 1, attr, stream);
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, g, bm, parts, len);
    if (e != cudaSuccess) return (int)e;
    VX_LAUNCH_CHECK();
    return VX_OK;
}

// Clusters of `blocks` blocks that run at once (a block fills an SM; clusters lie within a group of SMs: 33 of four, 15 of eight).
static int gt_clusters(int blocks, int sms) {
    static int cache[VX_MAX_DEVICES][GT_MAX_PARTS + 1];
    const int dev = vx_current_device();
    if (dev < 0) return sms / blocks;
    if (!cache[dev][blocks]) {
        static bool configured[VX_MAX_DEVICES];
        auto kernel = gemm_f32_tc_kernel<128, true, 1>;
        GtCall g = {};
        g.M = g.N = g.K = g.batch = 1;
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = gt_config<128>(g, 16, blocks, attr, nullptr);
        cfg.numAttrs = 1;   // (the cluster's size alone)
        int n = 0;
        if (vx_configure_smem(kernel, gt_smem(128) + 1024, configured) != VX_OK ||
            cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = sms / blocks;
        }
        cache[dev][blocks] = n;
    }
    return cache[dev][blocks];
}

template <int BM>
static int gt_go(const GtCall& g, bool vec, int per, int bm, int parts, int len, cudaStream_t stream) {
#define GT_GO(PER_) return vec ? gt_launch<BM, true, PER_>(g, bm, parts, len, stream) : gt_launch<BM, false, PER_>(g, bm, parts, len, stream)
    if (per == 1) GT_GO(1);
    if (per == 2) GT_GO(2);
    if (per == 4) GT_GO((BM <= 32 ? 4 : 2));
    GT_GO(0);
#undef GT_GO
}

// Row tiles (`bm` rows each), and whether and how the parts of k go to the blocks of a cluster (`per` parts a block, 0: no cluster): what takes
// the least time by the rounds of the SMs (of the clusters that run at once) and the time of a round, which was measured: a chunk takes 1.17 us
// and 4.5 ns a row up to 64 rows of A, 20 ns a row above; a round 2 us besides, with a cluster's sums 4 us and 10 ns a row.  Returns that time.
static double gt_plan(int M, int K, long long columns, int sms, int* best_bm, int* per) {
    int parts, len;
    gt_parts(K, &parts, &len);
    double best = 0;
    *best_bm = 0;
    for (int t = (M + 127) / 128; t <= (M + 127) / 128 + 3; ++t) {
        const int bm = ((M + t - 1) / t + 15) / 16 * 16;
        const long long tiles = columns * ((M + bm - 1) / bm);
        const double chunk = 1.17 + 0.0045 * bm + (bm > 64 ? 0.0155 * (bm - 64) : 0.0);
        for (int p = 0; p < parts && p <= (bm <= 32 ? 4 : 2); p = p ? 2 * p : 1) {   // (a cluster has two blocks or more)
            const int at_once = p ? gt_clusters((parts + p - 1) / p, sms) : sms, k = p ? p * len : K;
            const double cost = (double)((tiles + at_once - 1) / at_once) * ((p ? 4.0 + 0.01 * bm : 2.0) + chunk * ((k + GT_BK - 1) / GT_BK));
            if (!*best_bm || cost < best) { *best_bm = bm; *per = p; best = cost; }
        }
        if (bm <= 16) break;
    }
    return best;
}

// Whether a float32 product takes the tensor cores.  N and K alone say, because a row's result must not depend on how many rows the call has: a
// product that one call has for a decoded token another has for a prompt.  So they are taken where they are not slower for a few rows either: by
// estimates of both for eight rows, not by more than an eighth (the multiply-adds': a part's chain, 42 ns a k; 2.9 TB/s and 4.5 us).  Not for k
// below 1,024, where multiply-adds have short parts, nor for more than 32,768 columns, a vocabulary's head, of which a step wants a few rows.
// Measured, us, W from memory, multiply-adds and tensor cores (N x K), 8 rows: 4096 x 1024 10.9, 10.0; 6144 x 1024 14.8, 14.7; 1024 x 3072 14.0,
// 12.1; 4096 x 4096 28, 27.3; 4096 x 12288 74, 68; 12288 x 2048 40.9, 45.6; 24576 x 4096 122, 137; 2560 x 4096 22.2, 25.4; refused: 2048 x 2048
// 11.5, 14.2; 19456 x 2560 67.6, 88; 3072 x 512 5.1, 7.9; 8192 x 768 13.3, 14.8.
// 99 rows: 4096 x 1024 39, 17.7; 6144 x 1024 57, 26.2; 1024 x 3072 29.7, 21.3; 12288 x 2048 195, 90; 24576 x 4096 733, 284; 300 rows:
// 6144 x 1024 127, 43; 1024 x 2048 54, 25; 4096 x 12288 929, 390; (refused) 19456 x 2560 835, 355; 3072 x 512 37, 16.
extern "C" int vx_gemm_f32_takes_tc(int N, int K) {
    if (K < 1024 || N <= 0 || N > 32768) return 0;
    static int sms_cache[VX_MAX_DEVICES];
    int parts, len, bm, per;
    gt_parts(K, &parts, &len);
    const double chain = (long long)N * K < (6 << 20) ? 0.034 * len : 0.0425 * len, bytes = 4.5 + 4.0 * N * K / 2.9e6;
    return gt_plan(8, K, (N + GT_BN - 1) / GT_BN, vx_sm_count(sms_cache), &bm, &per) <= 1.125 * (chain > bytes ? chain : bytes);
}

int vx_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                   long long sa, long long sw, long long sc, int w_ready, int* error, cudaStream_t stream) {
    const GtCall g = {A, W, bias, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, w_ready, error};
    // rows that begin on 16-byte addresses are fetched 16 bytes at a time, others four
    const bool vec = !((lda | ldw) & 3) && !((sa | sw) & 3) && !((((uintptr_t)A) | ((uintptr_t)W)) & 15);
    static int sms_cache[VX_MAX_DEVICES];
    int parts, len, bm, per;
    gt_parts(K, &parts, &len);
    gt_plan(M, K, (long long)((N + GT_BN - 1) / GT_BN) * batch, vx_sm_count(sms_cache), &bm, &per);
    if ((M + bm - 1) / bm > 65535) return VX_ERR_LIMIT;
    if (bm <= 16) return gt_go<16>(g, vec, per, bm, parts, len, stream);
    if (bm <= 32) return gt_go<32>(g, vec, per, bm, parts, len, stream);
    if (bm <= 64) return gt_go<64>(g, vec, per, bm, parts, len, stream);
    return gt_go<128>(g, vec, per, bm, parts, len, stream);
}
