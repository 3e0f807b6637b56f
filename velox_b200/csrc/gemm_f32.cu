// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) in float32 on the CUDA cores: the matrix product of the 32-bit path
// where the tensor cores (gemm_f32_tc.cu) are slower for a few rows: a short k, a vocabulary's head, some sizes between.
//
// Order of a sum: k is cut into at most eight parts of equal length, by K alone (gf_parts); within a part the even and the
// odd k are summed apart, each in ascending order (two lanes of one packed multiply-add), then added; the parts' sums are
// added in ascending order.  Every configuration below keeps that order, so a row's result does not depend on how many rows
// the call has, and no multiply-add is wider or narrower than 32 bits.
//
// What bounds it: W's bytes for a few rows, the multiply-adds from some 40 rows on.  A and W come through a cp.async ring of
// [rows][32 k] tiles (rows padded to 36 floats: eight lanes that read 16 bytes of eight rows touch all banks once), a thread
// owns TM x TN outputs and reads four k of each of its rows with one load.  A product of few output tiles is cut along k as
// well: the parts go to the blocks of a cluster, which add them through distributed shared memory, so that a model of width
// 1,024 fills the chip (without: 16 to 64 blocks).  Measurements: at vx_gemm_f32 below.
#include <cooperative_groups.h>

#include "common.cuh"
#include "gemm_f32.cuh"

namespace cg = cooperative_groups;

#define GF32_BK 32
#define GF32_LD 36
#define GF32_STAGES 4
#define GF32_MAX_PARTS 8

__device__ __forceinline__ void gf_cp16(unsigned dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void gf_cp4(unsigned dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
// c.lo += a.lo b.lo, c.hi += a.hi b.hi: two 32-bit multiply-adds, each rounded by itself.
__device__ __forceinline__ void gf_fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float gf_halves(unsigned long long c) {
    return __uint_as_float((unsigned)c) + __uint_as_float((unsigned)(c >> 32));
}

// ROWS rows of X (from row r0 of `rows`) for k in [k0, k0 + 32), columns beyond `kend` and rows beyond the matrix as zeros.
template <int ROWS, int NT, bool VEC>
__device__ __forceinline__ void gf_load(float* dst, const float* __restrict__ X, int r0, int rows, int ld, int k0, int kend) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(dst);
    if (VEC) {
#pragma unroll 4
        for (int i = threadIdx.x; i < ROWS * 8; i += NT) {
            const int r = i >> 3, k = k0 + (i & 7) * 4;
            const bool in = r0 + r < rows && k < kend;
            gf_cp16(base + (r * GF32_LD + (i & 7) * 4) * 4, in ? X + (size_t)(r0 + r) * ld + k : X, in ? min(16, (kend - k) * 4) : 0);
        }
    } else {
        for (int i = threadIdx.x; i < ROWS * 32; i += NT) {
            const int r = i >> 5, k = k0 + (i & 31);
            const bool in = r0 + r < rows && k < kend;
            gf_cp4(base + (r * GF32_LD + (i & 31)) * 4, in ? X + (size_t)(r0 + r) * ld + k : X, in ? 4 : 0);
        }
    }
}

template <int TM, int TN, int TY, int TX, bool VEC, bool SPLIT>
__global__ void __launch_bounds__(TX* TY)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M,
                int N, int K, int lda, int ldw, int ldc, long long sa, long long sw, long long sc, int parts, int part_len, int w_ready) {
    constexpr int BM = TM * TY, BN = TN * TX, NT = TX * TY, STAGE = (BM + BN) * GF32_LD;
    extern __shared__ __align__(16) float gf_smem[];
    A += (size_t)blockIdx.z * sa;
    W += (size_t)blockIdx.z * sw;
    C += (size_t)blockIdx.z * sc;
    const int rank = SPLIT ? (int)blockIdx.x % parts : 0;
    const int n0 = (SPLIT ? (int)blockIdx.x / parts : (int)blockIdx.x) * BN, m0 = blockIdx.y * BM;
    const int kbeg = SPLIT ? rank * part_len : 0, kend = SPLIT ? min(K, kbeg + part_len) : K;
    const int chunks = (kend - kbeg + GF32_BK - 1) / GF32_BK;
    // eight neighbouring lanes read eight rows of W; the lanes of a warp share 4 (or fewer) rows of A
    constexpr int LX = TX < 8 ? TX : (TY >= 4 ? 8 : 32 / TY);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int WX = TX / LX;   // warps side by side
    const int tx = (warp % WX) * LX + lane % LX, ty = (warp / WX) * (32 / LX) + lane / LX;

    // a W that the caller calls ready depends on no earlier kernel: its first tiles are asked for before the wait
    if (!w_ready) pdl_wait();
#pragma unroll
    for (int s = 0; s < GF32_STAGES - 1; ++s)
        if (s < chunks) gf_load<BN, NT, VEC>(gf_smem + s * STAGE + BM * GF32_LD, W, n0, N, ldw, kbeg + s * GF32_BK, kend);
    pdl_wait();   // (a second time it returns at once)
    pdl_trigger();
#pragma unroll
    for (int s = 0; s < GF32_STAGES - 1; ++s) {
        if (s < chunks) gf_load<BM, NT, VEC>(gf_smem + s * STAGE, A, m0, M, lda, kbeg + s * GF32_BK, kend);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    unsigned long long acc[TM][TN];
    float total[SPLIT ? 1 : TM][SPLIT ? 1 : TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
    if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) total[SPLIT ? 0 : i][SPLIT ? 0 : j] = 0.f;
    }
    const int part_chunks = part_len / GF32_BK;
    int left = part_chunks;   // chunks until the part ends
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(GF32_STAGES - 2) : "memory");
        __syncthreads();   // (the tile of chunk c is there, and everyone is done with the one that is overwritten next)
        const int nx = c + GF32_STAGES - 1;
        if (nx < chunks) {
            float* st = gf_smem + (nx % GF32_STAGES) * STAGE;
            gf_load<BM, NT, VEC>(st, A, m0, M, lda, kbeg + nx * GF32_BK, kend);
            gf_load<BN, NT, VEC>(st + BM * GF32_LD, W, n0, N, ldw, kbeg + nx * GF32_BK, kend);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* as = gf_smem + (c % GF32_STAGES) * STAGE + ty * GF32_LD;
        const float* ws = gf_smem + (c % GF32_STAGES) * STAGE + (BM + tx) * GF32_LD;
#pragma unroll
        for (int k = 0; k < GF32_BK; k += 4) {
            ulonglong2 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + j * TX * GF32_LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * TY * GF32_LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    gf_fma2(acc[i][j], a.x, w[j].x);
                    gf_fma2(acc[i][j], a.y, w[j].y);
                }
            }
        }
        if (!SPLIT && (--left == 0 || c + 1 == chunks)) {
            left = part_chunks;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    total[SPLIT ? 0 : i][SPLIT ? 0 : j] += gf_halves(acc[i][j]);
                    acc[i][j] = 0ull;
                }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int m = m0 + ty + TY * i, n = n0 + tx + TX * j;
                if (m < M && n < N) C[(size_t)m * ldc + n] = total[SPLIT ? 0 : i][SPLIT ? 0 : j] + (bias ? bias[n] : 0.f);
            }
        return;
    }
    __syncthreads();   // (everyone is done with the ring, which now takes this part's sums)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) gf_smem[(ty + TY * i) * BN + tx + TX * j] = gf_halves(acc[i][j]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = rank * NT + threadIdx.x; e < BM * BN; e += parts * NT) {
        const int m = m0 + e / BN, n = n0 + e % BN;
        if (m >= M || n >= N) continue;
        float v = 0.f;
        for (int p = 0; p < parts; ++p) v += cluster.map_shared_rank(gf_smem, p)[e];
        C[(size_t)m * ldc + n] = v + (bias ? bias[n] : 0.f);
    }
    cluster.sync();   // (a block's sums are read until here)
}

// k's parts and their length (a multiple of 32), eight parts at most: of 256 k at least from 1,024 on, of 64 below, where the
// chains of a sum would else be as long as there (narrow models, whose errors nothing averages out).  No part is empty.
static void gf_parts(int K, int* parts, int* len) {
    int p = K / (K >= 1024 ? 256 : 64);
    p = p < 1 ? 1 : (p > GF32_MAX_PARTS ? GF32_MAX_PARTS : p);
    *len = ((K + p - 1) / p + GF32_BK - 1) / GF32_BK * GF32_BK;
    *parts = (K + *len - 1) / *len;
}

struct GfCall {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc, batch;
    long long sa, sw, sc;
    int w_ready;
};

template <int TM, int TN, int TY, int TX, bool VEC, bool SPLIT>
static int gf_launch(const GfCall& g, int parts, int len, cudaStream_t stream) {
    constexpr int BM = TM * TY, BN = TN * TX;
    auto kernel = gemm_f32_kernel<TM, TN, TY, TX, VEC, SPLIT>;
    size_t smem = (size_t)GF32_STAGES * (BM + BN) * GF32_LD * sizeof(float);
    static_assert(GF32_STAGES * (BM + BN) * GF32_LD >= BM * BN, "a part's sums fit into the ring");
    static bool configured[VX_MAX_DEVICES];
    if (int rc = vx_configure_smem(kernel, smem, configured)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.N + BN - 1) / BN * (SPLIT ? parts : 1)), (unsigned)((g.M + BM - 1) / BM), (unsigned)g.batch);
    cfg.blockDim = dim3(TX * TY);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (vx_pdl_is_enabled() && ((vx_pdl_mask() >> VX_K_GEMM) & 1)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (SPLIT) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = parts;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, g.A, g.W, g.bias, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc, g.sa, g.sw, g.sc, parts, len,
                                       g.w_ready);
    if (e != cudaSuccess) return (int)e;
    VX_LAUNCH_CHECK();
    return VX_OK;
}

static long long gf_tiles(const GfCall& g, int bm, int bn) {
    return (long long)((g.N + bn - 1) / bn) * ((g.M + bm - 1) / bm) * g.batch;
}

template <int TM, int TN, int TY, int TX>
static int gf_choose(const GfCall& g, bool vec, bool whole, cudaStream_t stream) {
    int parts, len;
    gf_parts(g.K, &parts, &len);
    if (parts > 1 && !whole)
        return vec ? gf_launch<TM, TN, TY, TX, true, true>(g, parts, len, stream) : gf_launch<TM, TN, TY, TX, false, true>(g, parts, len, stream);
    return vec ? gf_launch<TM, TN, TY, TX, true, false>(g, parts, len, stream) : gf_launch<TM, TN, TY, TX, false, false>(g, parts, len, stream);
}

// Which tile (measured, microseconds; before: the 64 x 64 tile with scalar loads that took every size):
//   rows x N x K         before   8 x 64   16 x 64   32 x 64   64 x 64
//   1 x 4096 x 1024        71       11.3     10.4      13.6      25.6
//   8 x 2560 x 9728       797       48.3     55.1      84.6     113.6
//   24 x 4096 x 1024       78        -        -        14.8      26.3
//   99 x 1024 x 2048      119        -        -        21.3      26.7
//   99 x 4096 x 1024       77        -        -        41.8      38.0
//   2000 x 4096 x 1024    628        -        -       475       430
// Tiles of 64 rows x 128 columns and of 128 x 128 (8 x 8 outputs a thread) were tried: 36 to 47 microseconds where these
// take 21 to 38, and no faster at 2,000 rows.  Error against 64 bits at K = 1024 / 3072 / 9728: 2.1e-7 / 2.6e-7 / 4.5e-7 (before, one
// ascending sum: 5.7e-7 / 9.9e-7 / 1.8e-6).
// Whether the parts of k go to the blocks of a cluster: not where there are tiles enough without.  Up to 32 rows that takes 8 tiles an SM
// (151,936 columns, one row: 162 whole, 181 cut; 4096 x 1024: 38 and 11), above, with tiles of 64 rows, 2.5 (rows x N x K,
// whole and cut: 150 x 8192 x 2048 197 and 201; 1000 x 4096 x 512 114 and 183; at 2.2 tiles an SM 300 x 4096 x 2048 197 and 170).
// Below k = 1,024, where a part is short against the cluster's barriers, less: whole from K / 170 tiles of 32 rows an SM on, as these as long as
// four an SM hold them all, else as tiles of 64 rows (whole, and cut in the better of the two tiles): 128 x 4096 x 128 7.7 and 9.3 to 11.8;
// 128 x 8192 x 256 19.3 and 28.7 (the kernel before these: 25.2); 300 x 4096 x 256 26.6 and 33; 150 x 2048 x 256 12.7 and 11.7, cut; 128 x 8192 x 512
// 37 and 50; 300 x 2048 x 512 37 and 32, cut.  Rows that begin on no 16-byte address wait for their loads and are cut longer: 128 x 8192 x
// 1001 129 and 102 (the kernel before these: 94, the one size at which it is ahead).
int vx_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                long long sa, long long sw, long long sc, int w_ready, cudaStream_t stream) {
    const GfCall g = {A, W, bias, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, w_ready};
    // rows that begin on 16-byte addresses are fetched 16 bytes at a time, others four
    const bool vec = !((lda | ldw) & 3) && !((sa | sw) & 3) && !((((uintptr_t)A) | ((uintptr_t)W)) & 15);
    static int sms_cache[VX_MAX_DEVICES];
    const long long sms = vx_sm_count(sms_cache);
    if (M <= 4 && gf_tiles(g, 4, 128) >= 8 * sms) return gf_choose<4, 4, 1, 32>(g, vec, true, stream);   // (143 against 162 microseconds there)
    // up to 8 rows: the wide rows pay where W is large
    if (M <= 8 && (long long)N * K >= (6 << 20)) return gf_choose<8, 2, 1, 32>(g, vec, gf_tiles(g, 8, 64) >= 8 * sms, stream);
    if (M <= 16) return gf_choose<4, 4, 4, 16>(g, vec, gf_tiles(g, 16, 64) >= 8 * sms, stream);
    int parts, len;
    gf_parts(K, &parts, &len);
    const long long t32 = gf_tiles(g, 32, 64), t64 = gf_tiles(g, 64, 64);
    if (M <= 32) return gf_choose<8, 4, 4, 16>(g, vec, t32 >= 8 * sms, stream);
    // a narrow k: the parts are short against the cluster's barriers, the shorter the fewer tiles it takes to do without
    if (K <= 128 || (vec && K < 1024 && t32 * 170 >= K * sms))
        return t32 <= 4 * sms ? gf_choose<8, 4, 4, 16>(g, vec, true, stream) : gf_choose<8, 4, 8, 16>(g, vec, true, stream);
    if (t32 * parts <= 4 * sms) return gf_choose<8, 4, 4, 16>(g, vec, false, stream);
    return gf_choose<8, 4, 8, 16>(g, vec, 2 * t64 >= 5 * sms, stream);
}
