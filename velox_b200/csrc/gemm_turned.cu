// C[M,N] = A[M,K] * W[N,K]^T in bfloat16 on the fifth-generation tensor cores with the operands turned: out^T = W A^T, rows of W on
// the M side of tcgen05.mma, rows of A as its columns.  For products of 9 to some hundred rows.
//
// The M side of an instruction is 128 rows (256 by a pair of blocks), the other any multiple of 16: with A's rows there a product of
// 20 rows wastes nothing on padding, and one of 312 takes columns for just so many.
//
// A tile is 128 CG rows of W by n rows of A (CG 1: a block; CG 2: a pair of blocks, `cta_group::2`, each of which brings its
// 128 rows of W and half of the rows of A; nothing is multicast).  K may be cut into `splits` runs, one to each block (or pair) of a cluster, whose
// float32 sums are added in ascending order through distributed shared memory.  The W tiles from `full_w` on may have narrower tiles
// (n2 rows of A): where the tiles would begin a round of the SMs that they cannot fill, that round's work is spread over all of them.
// Warps of a block:
//   warp 0    producer: asks for W's first stages before it waits for the kernel launched before this one (if the caller says
//             that W is ready), for A's after, then for stage after stage, through all of the block's tiles (persistent blocks);
//   warp 1    tensor memory; (in the leading block) issues the products;
//   warps 2-9 epilogue: lanes are rows of W, so gate and up rows (tiles of 8 + 8) are eight lanes apart and a warp's stores run along
//             the rows of C; two accumulators, so that a tile's epilogue runs under the next one's products.
// Every wait on an mbarrier is bounded; a block whose wait runs out records a code in the caller's error word and writes NaN, the others
// run out of theirs, all meet at the cluster's barrier, free their tensor memory and return.
//
// Tensor memory is taken before the wait for the kernel before: of the kernels that take some only this one, with two blocks an
// SM, leaves room for a block beside its own, and it lets the next kernel in after it has taken its own.
//
// What bounds it: W's bytes up to some 64 rows, above that what the SMs can fetch from L2 (80 to 120 bytes a ns and SM) before the
// tensor cores.  Measurements and the choice of a tile: at gu_plan below.
//
// Sizes: K a multiple of 8, rows of A, W and C 16-byte aligned, N a multiple of 16.
#include "tcgen05_pair.cuh"

#define GU_THREADS 320
#define GU_EPI_WARPS 8
#define GU_MAX_STAGES 12
#define GU_ERR_PRODUCER 7
#define GU_ERR_MMA 8
#define GU_ERR_EPILOGUE 9
#define GU_W_BYTES (128 * TC_BK * 2)

struct GuShape {
    int n;              // rows of A in a tile: an instruction's columns
    int splits;         // runs of k
    int full_w, n2;     // W tiles from full_w on take tiles of n2 rows of A (n2 0: none do)
    int stages;         // of the ring
    int kbs;            // k blocks of a run
};

__device__ __forceinline__ void gu_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float2 gu_ld_cluster2(unsigned addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float gu_ld_cluster(unsigned addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void gu_put2(bf16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }
__device__ __forceinline__ void gu_put2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }

template <int CG, bool GATED, typename TO>
__global__ void __launch_bounds__(GU_THREADS)
gemm_turned_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_x2,
                   TO* __restrict__ C, int M, int N, int K, int ldc, int act, int w_ready, const GuShape sh, int* __restrict__ error) {
    extern __shared__ unsigned char gu_raw[];
    __shared__ __align__(8) unsigned long long full_bar[GU_MAX_STAGES], empty_bar[GU_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_s;
    unsigned char* tiles = (unsigned char*)(((uintptr_t)gu_raw + 1023) & ~(uintptr_t)1023);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const unsigned crank = tp_cluster_rank();        // (0 without a cluster)
    const unsigned rank = CG == 2 ? crank & 1 : 0, lead = CG == 2 ? crank & ~1u : crank;
    const int team = CG * sh.splits;                 // blocks that form a tile
    const int split = sh.splits > 1 ? (int)crank / CG : 0;
    const unsigned stage_bytes = GU_W_BYTES + (unsigned)(sh.n / CG) * (TC_BK * 2);
    const unsigned tmem_cols = 2 * sh.n <= 32 ? 32 : (1u << (32 - __clz(2 * sh.n - 1)));
    const int nkb_all = (K + TC_BK - 1) / TC_BK, kb0 = split * sh.kbs, nkb = min(nkb_all - kb0, sh.kbs);
    const int xt1 = (M + sh.n - 1) / sh.n, xt2 = sh.n2 ? (M + sh.n2 - 1) / sh.n2 : 1;
    const int wtiles = (N + 128 * CG - 1) / (128 * CG);
    const int main_tiles = sh.full_w * xt1, total = main_tiles + (wtiles - sh.full_w) * xt2;
    const int me = (int)blockIdx.x / team, teams = (int)gridDim.x / team;
    const int my_tiles = (total - me + teams - 1) / teams;
    struct Tile { int w0, m0, n; };
    // tiles that are worked on at the same time share a tile of W
    auto tile_of = [&](int ti) {
        const int t = me + ti * teams;
        if (t < main_tiles) return Tile{(t / xt1) * 128 * CG + (int)rank * 128, (t % xt1) * sh.n, sh.n};
        const int u = t - main_tiles;
        return Tile{(sh.full_w + u / xt2) * 128 * CG + (int)rank * 128, (u % xt2) * sh.n2, sh.n2};
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < sh.stages; ++s) {
            tc_mbar_init(tc_smem_u32(&full_bar[s]), 1);    // the leading block's producer (with the bytes of both)
            tc_mbar_init(tc_smem_u32(&empty_bar[s]), 1);   // the commit of the products that read the stage
        }
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(tc_smem_u32(&acc_full[i]), 1);
            tc_mbar_init(tc_smem_u32(&acc_empty[i]), GU_EPI_WARPS * CG);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_s)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_s)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    if (CG == 2) tp_cluster_sync();   // (the other block's mbarriers and tensor memory are there before anything is written to them)
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = tmem_s;

    // ---- producer's loads: stage s, k block kb ----
    auto load = [&](const Tile& t, int kb, int s, bool of_w, bool of_x) {
        const unsigned bar = tc_smem_u32(&full_bar[s]), st = tc_smem_u32(tiles) + (unsigned)s * stage_bytes;
        const int xrows = t.n / CG, k = (kb0 + kb) * TC_BK;
        const unsigned lead_bar = CG == 2 ? tp_map_to_rank(bar, lead) : bar;
        if (of_w) {
            if (rank == 0) tc_mbar_expect_tx(bar, CG * (GU_W_BYTES + (unsigned)xrows * (TC_BK * 2)));
            if (CG == 2) tp_tma_load_2d(st, &map_w, k, t.w0, lead_bar);
            else tc_tma_load_2d(st, &map_w, k, t.w0, bar);
        }
        if (of_x) {
            const CUtensorMap* map = t.n == sh.n ? &map_x : &map_x2;
            const int row = t.m0 + (int)rank * xrows;
            if (CG == 2) tp_tma_load_2d(st + GU_W_BYTES, map, k, row, lead_bar);
            else tc_tma_load_2d(st + GU_W_BYTES, map, k, row, bar);
        }
    };
    const int ahead = w_ready ? min(sh.stages, nkb) : 0;   // stages whose W is asked for before the wait
    if (warp == 0 && ahead) {
        const Tile t = tile_of(0);
        for (int kb = 0; kb < ahead; ++kb)
            if (tc_elect()) load(t, kb, kb, true, false);
    }
    pdl_wait();
    if (warp == 0 && ahead) {
        const Tile t = tile_of(0);
        for (int kb = 0; kb < ahead; ++kb)
            if (tc_elect()) load(t, kb, kb, false, true);
    }
    __syncwarp();
    pdl_trigger();

    if (warp == 0) {
        int s = ahead == sh.stages ? 0 : ahead;
        unsigned phase = ahead == sh.stages ? 0 : 1;   // (the first time round a stage is free: the phase before the first has ended)
        for (int ti = 0; ti < my_tiles; ++ti) {
            const Tile t = tile_of(ti);
            for (int kb = ti ? 0 : ahead; kb < nkb; ++kb) {
                if (!tc_warp_wait(tc_smem_u32(&empty_bar[s]), phase)) {
                    if (lane == 0) atomicExch(error, GU_ERR_PRODUCER);
                    ti = my_tiles;
                    break;
                }
                if (tc_elect()) load(t, kb, s, true, true);
                if (++s == sh.stages) { s = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            int s = 0;
            unsigned phase = 0;
            bool ok = true;
            for (int ti = 0; ok && ti < my_tiles; ++ti) {
                const Tile t = tile_of(ti);
                // float32 accumulator, bfloat16 operands, both K-major, N = n, M = 128 CG
                const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(t.n >> 3) << 17) | ((unsigned)(128 * CG >> 4) << 24);
                const int buf = ti & 1, use = ti >> 1;
                const unsigned d = tmem + (unsigned)(buf * sh.n);
                // the epilogue must have emptied this accumulator
                ok = !use || tc_warp_wait(tc_smem_u32(&acc_empty[buf]), (unsigned)((use - 1) & 1));
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                for (int kb = 0; ok && kb < nkb; ++kb) {
                    ok = tc_warp_wait(tc_smem_u32(&full_bar[s]), phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const unsigned wd = tc_desc_lo(tc_smem_u32(tiles) + (unsigned)s * stage_bytes);
                    if (tc_elect()) {
                        tc_mma_run<CG, TC_BK / 16>(d, wd, wd + (GU_W_BYTES >> 4), idesc, kb > 0);
                        if (CG == 2) tp_commit_mask(tc_smem_u32(&empty_bar[s]), (unsigned short)(3u << lead));
                        else tc_commit(tc_smem_u32(&empty_bar[s]));
                    }
                    if (++s == sh.stages) { s = 0; phase ^= 1; }
                }
                if (ok && tc_elect()) {
                    if (CG == 2) tp_commit_mask(tc_smem_u32(&acc_full[buf]), (unsigned short)(3u << lead));
                    else tc_commit(tc_smem_u32(&acc_full[buf]));
                }
            }
            if (!ok && lane == 0) atomicExch(error, GU_ERR_MMA);
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const int l = quarter * 32 + lane;   // this thread's row of the block's 128 rows of W
        bool ok = true;
        for (int ti = 0; ti < my_tiles; ++ti) {
            const Tile t = tile_of(ti);
            const int buf = ti & 1, use = ti >> 1;
            if (ok) {
                ok = tc_warp_wait(tc_smem_u32(&acc_full[buf]), (unsigned)(use & 1));
                if (!ok && lane == 0) atomicExch(error, GU_ERR_EPILOGUE);
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned acc = tmem + (unsigned)(buf * sh.n) + ((unsigned)(quarter * 32) << 16);
            const int width = min(t.n, M - t.m0);   // (columns that are rows of A)
            const bool mine = t.w0 + quarter * 32 + (lane & ~15) < N;   // (N is a multiple of 16)
#pragma unroll 1
            for (int c0 = half * 16; c0 < width; c0 += 32) {
                unsigned r[16];
                if (ok) {
                    gu_ld16(acc + (unsigned)c0, r);
                } else {   // (a wait ran out, and the error word says so: NaN rather than what the memory held)
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = 0x7fc00000u;
                }
                if (sh.splits > 1) {
                    float* sums = reinterpret_cast<float*>(tiles);   // [n][128], in place of the stages
#pragma unroll
                    for (int j = 0; j < 16; ++j) sums[(c0 + j) * 128 + l] = __uint_as_float(r[j]);
                } else if (GATED) {
                    // of two columns the lanes of gate rows take the first, those of up rows the second
                    const bool up = lane & 8;
                    const int f = ((t.w0 + l) >> 4) * 8 + (lane & 7);
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const float a = __uint_as_float(r[j]), b = __uint_as_float(r[j + 1]);
                        const float o = __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
                        const float v = activation(up ? o : a, act) * (up ? b : o);
                        const int c = c0 + j + (up ? 1 : 0);
                        if (mine && c < width) C[(size_t)(t.m0 + c) * ldc + f] = from_f32<TO>(v);
                    }
                } else if (sizeof(TO) == 4) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (mine && c0 + j < width) C[(size_t)(t.m0 + c0 + j) * ldc + t.w0 + l] = from_f32<TO>(__uint_as_float(r[j]));
                } else {
                    // of two columns the even lanes take the first, with their neighbour's row beside theirs
                    const bool odd = lane & 1;
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const float a = __uint_as_float(r[j]), b = __uint_as_float(r[j + 1]);
                        const float o = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
                        const int c = c0 + j + (odd ? 1 : 0);
                        if (mine && c < width) gu_put2(C + (size_t)(t.m0 + c) * ldc + t.w0 + (l & ~1), odd ? o : a, odd ? b : o);
                    }
                }
            }
            // the accumulator may be overwritten once the epilogue warps (of both blocks) have read it
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) tp_arrive_remote(tp_map_to_rank(tc_smem_u32(&acc_empty[buf]), lead));
                else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem_u32(&acc_empty[buf])) : "memory");
            }
        }
    }
    // All blocks of a team meet before the tensor memory goes back: the leading block's products read the other's shared memory and
    // arrive on its mbarriers (every wait above was bounded); and a split's sums are all there.
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    if (CG == 2 || sh.splits > 1) tp_cluster_sync();
    else __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
    if (sh.splits > 1) {
        // each block of the team adds its share of the columns, run after run
        const Tile t = tile_of(0);
        const int width = min(sh.n, M - t.m0), c_end = min(width, (split + 1) * sh.n / sh.splits), c_beg = min(width, split * sh.n / sh.splits);
        const unsigned base = tc_smem_u32(tiles);
        for (int e = (int)threadIdx.x; e < (c_end - c_beg) * 64; e += GU_THREADS) {
            const int c = c_beg + (e >> 6), i = e & 63;
            const int row = GATED ? (i >> 3) * 16 + (i & 7) : 2 * i;
            if (t.w0 + row >= N) continue;
            float a = 0.f, b = 0.f;
            for (int p = 0; p < sh.splits; ++p) {
                const unsigned at = tp_map_to_rank(base + (unsigned)(c * 128 + row) * 4, (unsigned)(p * CG) + rank);
                if (GATED) {
                    a += gu_ld_cluster(at);
                    b += gu_ld_cluster(at + 32);
                } else {
                    const float2 v = gu_ld_cluster2(at);
                    a += v.x;
                    b += v.y;
                }
            }
            TO* dst = C + (size_t)(t.m0 + c) * ldc;
            if (GATED) dst[((t.w0 + row) >> 4) * 8 + (row & 7)] = from_f32<TO>(activation(a, act) * b);
            else gu_put2(dst + t.w0 + row, a, b);
        }
        __syncwarp();
        tp_cluster_sync();   // (a block's sums are read until here)
    }
}

// ---- host side ----
template <int CG, bool GATED, typename TO>
static int gu_launch(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mx2, TO* C, int M, int N, int K, int ldc, int act, int w_ready,
                     const GuShape& sh, size_t smem, int teams, int* error, cudaStream_t stream) {
    auto kernel = gemm_turned_kernel<CG, GATED, TO>;
    static bool configured[VX_MAX_DEVICES];
    if (int rc = vx_configure_smem(kernel, 226 * 1024, configured)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(teams * CG * sh.splits));
    cfg.blockDim = dim3(GU_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (vx_pdl_is_enabled() && ((vx_pdl_mask() >> VX_K_GEMM) & 1)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (CG * sh.splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = CG * sh.splits;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, mw, mx, mx2, C, M, N, K, ldc, act, w_ready, sh, error);
    if (e != cudaSuccess) return (int)e;
    VX_LAUNCH_CHECK();
    return VX_OK;
}

// With a tile's shape: cg 1 or 2; n a multiple of 16 up to 256 (128 with two blocks an SM); splits with cg * splits <= 8; n2 and full_w
// as above (without splits); per_sm 1 or 2 blocks an SM.  gated: W's rows come in tiles of 8 gate rows followed by their 8 up rows and C is
// [M, N/2] = act(gate) * up.  `w_ready`: W is not something the kernel launched just before this one writes.
extern "C" int vx_gemm_turned_shape(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int gated, int act,
                                    int out_dtype, int w_ready, int cg, int n, int splits, int full_w, int n2, int per_sm,
                                    int* error, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return VX_OK;
    if (K <= 0 || (K & 7) || (N & 15) || !error || gated < 0 || gated > 1 || (gated && (act < 0 || act > VX_ACT_LAST))) return VX_ERR_SHAPE;
    if ((lda & 7) || (ldw & 7) || (ldc & 7) || lda < K || ldw < K) return VX_ERR_ALIGN;
    if ((((uintptr_t)A) | ((uintptr_t)W) | ((uintptr_t)C)) & 15) return VX_ERR_ALIGN;
    if (ldc < (gated ? N / 2 : N)) return VX_ERR_SHAPE;
    if (out_dtype != VX_BF16 && out_dtype != VX_F32) return VX_ERR_DTYPE;
    if (cg < 1 || cg > 2 || per_sm < 1 || per_sm > 2 || n < 16 || n > 256 / per_sm || (n & 15) || splits < 1 || cg * splits > 8) return VX_ERR_SHAPE;
    const int wtiles = (N + 128 * cg - 1) / (128 * cg), nkb = (K + TC_BK - 1) / TC_BK;
    if (splits > nkb || (n2 && (splits > 1 || n2 < 16 || n2 > n || (n2 & 15) || full_w < 0 || full_w > wtiles))) return VX_ERR_SHAPE;
    GuShape sh;
    sh.n = n;
    sh.kbs = (nkb + splits - 1) / splits;
    sh.splits = (nkb + sh.kbs - 1) / sh.kbs;   // (no run is empty)
    sh.full_w = n2 ? full_w : wtiles;
    sh.n2 = n2;
    const int stage = GU_W_BYTES + n / cg * (TC_BK * 2);
    // (with one block an SM the ring leaves no room for a block of another tcgen05 product beside it; the sums of a split fit into it)
    const int stages = (per_sm == 2 ? 108 * 1024 : 221 * 1024) / stage;
    sh.stages = stages > GU_MAX_STAGES ? GU_MAX_STAGES : stages;
    if (sh.stages < 2 || (sh.splits > 1 && sh.stages * stage < n * 512)) return VX_ERR_SHAPE;
    const size_t smem = (size_t)sh.stages * stage + 1024;
    CUtensorMap mw, mx, mx2;
    if (!tc_make_map(&mw, W, N, K, ldw, 128) || !tc_make_map(&mx, A, M, K, lda, n / cg)) return VX_ERR_DRIVER;
    mx2 = mx;
    if (n2 && n2 != n && !tc_make_map(&mx2, A, M, K, lda, n2 / cg)) return VX_ERR_DRIVER;
    static int sm_counts[VX_MAX_DEVICES];
    const int sms = vx_sm_count(sm_counts);
    const long long tiles = (long long)sh.full_w * ((M + n - 1) / n) + (long long)(wtiles - sh.full_w) * (n2 ? (M + n2 - 1) / n2 : 1);
    if (tiles > 0x7fffff) return VX_ERR_LIMIT;
    const int slots = sms * per_sm / cg;
    const int teams = sh.splits > 1 ? (int)tiles : (int)(tiles < slots ? tiles : slots);
#define GU_GO(CG_, G_, T_) gu_launch<CG_, G_, T_>(mw, mx, mx2, (T_*)C, M, N, K, ldc, act, w_ready, sh, smem, teams, error, stream)
    if (out_dtype == VX_BF16) {
        if (cg == 2) return gated ? GU_GO(2, true, bf16) : GU_GO(2, false, bf16);
        return gated ? GU_GO(1, true, bf16) : GU_GO(1, false, bf16);
    }
    if (cg == 2) return gated ? GU_GO(2, true, float) : GU_GO(2, false, float);
    return gated ? GU_GO(1, true, float) : GU_GO(1, false, float);
#undef GU_GO
}

// Clusters of `blocks` blocks, each of which fills an SM, that run at once (a cluster lies within a group of SMs).  A plan that counted on 18
// clusters of seven had some of 16 wait for the others: 150 x 2048 x 6144 22.8 us, in the six runs that are chosen now 13.5.
static int gu_clusters(int blocks, int sms) {
    static int cache[VX_MAX_DEVICES][9];
    const int dev = vx_current_device();
    if (dev < 0) return sms / blocks;
    int& n = cache[dev][blocks];
    if (!n) {
        static bool configured[VX_MAX_DEVICES];
        auto kernel = gemm_turned_kernel<1, false, bf16>;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = blocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(blocks * sms));
        cfg.blockDim = dim3(GU_THREADS);
        cfg.dynamicSmemBytes = 222 * 1024;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int found = 0;
        if (vx_configure_smem(kernel, 226 * 1024, configured) != VX_OK || cudaOccupancyMaxActiveClusters(&found, kernel, &cfg) != cudaSuccess || found <= 0) {
            cudaGetLastError();
            found = sms / blocks;
        }
        n = found;
    }
    return n;
}

struct GuPlan { int cg, n, splits, full_w, n2, per_sm; };
static int gu_up16(int x) { return (x + 15) & ~15; }

// The tile, from measurements (us, kernel alone, W from memory).
// Up to 64 rows all rows of A are one tile and what counts is that W streams through all SMs:
//   120 W tiles and more: two blocks an SM (24 x 24576 x 4096 gated 35.3, one block 38.2; the library and the activation's kernel 39.0);
//   80 to 119: one block an SM up to 32 rows (24 x 12288 x 2048 13.0), else two row tiles, two blocks an SM (64 rows 13.3; 14.2 whole);
//   fewer: k in runs, as many as make 256 blocks, two an SM (24 x 2560 x 4096: 8 runs 7.3, 4 8.4, library 8.6); runs of 8 k blocks at least,
//   of 4 where there would not be 64 blocks; from 48 rows on with a long k one block an SM (64 x 2560 x 9728: 6 runs 13.4, 8 runs two an SM 14.4).
// Above, the least time by rounds of the SMs: a k block takes 0.10 us + 1.1 ns a row of A by pairs, 0.12 + 1.2 by single blocks, 0.24 + 2 with
// two an SM; 4.5 us besides, 2.2 for adding runs (measured and so: 312 x 19456 x 2560 gated 33.6, 32.0; 777 x 24576 x 4096 gated 124, 124;
// 312 x 2560 x 9728 19.9, 20.8; 150 x 12288 x 2048 gated 16.4, 16.3).
static GuPlan gu_plan(int M, int N, int K, int sms) {
    const int w1 = (N + 127) / 128, nkb = (K + TC_BK - 1) / TC_BK;
    if (M <= 64) {
        const int n = gu_up16(M);
        if (w1 >= 120) return GuPlan{1, n, 1, w1, 0, 2};
        if (w1 >= 80) return M <= 32 ? GuPlan{1, n, 1, w1, 0, 1} : GuPlan{1, 32, 1, w1, 0, 2};
        int s = 256 / w1, most = nkb / 8;
        const int few = nkb / 4 < 64 / w1 ? nkb / 4 : 64 / w1;
        if (most < few) most = few;
        int per_sm = 2;
        if (n >= 48 && nkb >= 64 && 130 / w1 >= 4) { s = 130 / w1 < 6 ? 130 / w1 : 6; per_sm = 1; }
        s = s < most ? s : most;
        s = s < 1 ? 1 : (s > 8 ? 8 : s);
        return GuPlan{1, n, s, w1, 0, per_sm};
    }
    GuPlan best = {};
    double least = 0;
    auto consider = [&](const GuPlan& p, double cost) {
        if (!best.cg || cost < least) { best = p; least = cost; }
    };
    for (int x = 1; x <= 8 || !best.cg; ++x) {
        const int n = gu_up16((M + x - 1) / x);
        if (n > 256 || (M + n - 1) / n != x) continue;
        for (int kind = 0; kind < 3; ++kind) {   // single blocks, two an SM, pairs
            const int cg = kind == 2 ? 2 : 1, per_sm = kind == 1 ? 2 : 1;
            if (per_sm == 2 && n > 128) continue;
            const int w = (N + 128 * cg - 1) / (128 * cg), slots = sms * per_sm / cg, tiles = w * x;
            auto block = [&](int rows) { return kind == 2 ? 0.10 + 0.0011 * rows : (kind == 1 ? 0.24 + 0.002 * rows : 0.12 + 0.0012 * rows); };
            consider(GuPlan{cg, n, 1, w, 0, per_sm}, 4.5 + (double)((tiles + slots - 1) / slots) * nkb * block(n));
            const int full = tiles / slots * slots / x;   // W tiles of the whole rounds
            if (per_sm == 1 && full > 0 && full < w)
                for (int n2 = 16; n2 <= 96 && n2 < n; n2 += n2 < 32 ? 16 : 32) {
                    const int rest = (w - full) * ((M + n2 - 1) / n2);
                    consider(GuPlan{cg, n, 1, full, n2, 1}, 4.5 + nkb * ((double)((full * x + slots - 1) / slots) * block(n) + (double)((rest + slots - 1) / slots) * block(n2)));
                }
            if (per_sm == 1)
                for (int s = 2; s * cg <= 8 && nkb / s >= 8; ++s) {
                    if (tiles > gu_clusters(s * cg, sms)) break;
                    consider(GuPlan{cg, n, s, w, 0, 1}, 6.7 + ((nkb + s - 1) / s) * block(n));
                }
        }
    }
    return best;
}

// The product with the tile that gu_plan gives; the arguments as above.
extern "C" int vx_gemm_turned(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int gated, int act,
                              int out_dtype, int w_ready, int* error, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return VX_OK;
    if (K <= 0) return VX_ERR_SHAPE;
    static int sm_counts[VX_MAX_DEVICES];
    const GuPlan p = gu_plan(M, N, K, vx_sm_count(sm_counts));
    return vx_gemm_turned_shape(A, W, C, M, N, K, lda, ldw, ldc, gated, act, out_dtype, w_ready, p.cg, p.n, p.splits, p.full_w, p.n2, p.per_sm,
                                error, stream);
}

// Whether a step's product of M rows with a model's weights is fastest this way, with its neighbours in the step: the kernels before and
// after it overlap it (programmatic launch), which they don't with the library's product.
// Measured in steps of 12 layers (us a step: without it and with it, everything else the same; shapes of 0.6B, 1.7B, 4B and 8B, whose gated products
// have N = 6,144, 12,288, 19,456 and 24,576 and whose deep ones 1,024 x 3072, 2,048 x 6144, 2,560 x 9728 and 4,096 x 12288):
//   9 to 32 rows   all products: 9 rows 643, 527; 733, 734; 1,025, 955; 1,437, 1,361; 32 rows 741, 694; 863, 855; 1,118, 1,075; 1,539, 1,492.
//   33 to 64 rows  wide gated and large deep ones.  For the others what they gain is less than what the host's wait for the step costs, which the
//                  library's products do without: 64 rows, none at all 829, all 956 (0.6B); 1,042, 1,079 (1.7B); alone 64 x 6144 x 2560 9.2 us, 13.0.
//   gated, above   up to 400 rows for N below 8,192 (150 rows 1,123, 1,041; 777 alone 18.9 us, 21.0), 640 below 16,384 (400 rows 1,369, 1,315; 512
//                  1,430, 1,425; 720 1,610, 1,629), else 800 (4B 312 rows 1,667, 1,577; 760 2,543, 2,485; 850 2,752, 2,744).  Not 225 to 256 rows
//                  of the middle ones, which are two whole tiles of gemm_tcgen05 (1,202, 1,240; 264 rows 1,240, 1,183).
//   deep (K of 2 N and more), above   up to 320 rows: 70 rows 1,141, 1,108 (1.7B); 150 rows 1,395, 1,353 (4B); 200 rows 2,082, 1,964 (8B); 312 rows
//                  1,664, 1,577 (4B); 328 1,676, 1,669; 360 1,682, 1,696.  Not 225 to 256 rows, whole tiles of the library's (1,481, 1,513; 1,990, 2,051),
//                  nor, for N of 2,048, more than 192 (208 rows 1,162, 1,181; 312 1,204, 1,221); but of smaller ones, whose steps wait for the
//                  host's launches (256 rows 1,139, 1,053).
// Where more than 64 rows are there a step has a prompt's attention, whose waits the host waits for anyway.
extern "C" int vx_gemm_turned_wins(int M, int N, int K, int gated) {
    if (M <= 8 || N <= 0 || K <= 0 || (N & 15) || (K & 7) || (!gated && N > 32768)) return 0;
    if (M <= 32) return 1;
    const bool whole = M > 224 && M <= 256;
    if (gated) return N >= 16384 ? M <= 800 : (M > 64 && (N >= 8192 ? M <= 640 && !whole : M <= 400));
    return K >= 2 * N && (M <= 64 ? N >= 2560 : (N < 2048 ? M <= 320 : (N < 2560 ? M <= 192 : M <= 320 && !whole)));
}
