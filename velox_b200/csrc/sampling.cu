// Token sampling from float32 logits: greedy, temperature, temperature + top-p.
//
// A cluster of one to eight blocks per row, as many as let all rows' clusters run at once.  For row r with temperature T, nucleus mass P and a
// uniform number u in [0,1) that the host drew for this (request, step):
//   T <= 1e-7:  the argmax, the lowest index winning ties.
//   otherwise:  e_i = 2^((x_i - max) log2(e) / T);  with 0 < P < 1 only the most
//               likely tokens stay whose mass reaches P (the one that crosses P and
//               its ties included): the kept tokens are those with e_i >= the largest
//               float t whose mass {e >= t} still reaches P times the whole;  the token
//               is the first index, in index order, whose cumulative kept mass
//               exceeds u times the kept total.
// Each block reads its part of the row once, all loads in flight together, and keeps it in shared memory (where it fits)
// when it is needed again; maxima, histograms and masses are put together through the cluster's shared memory, where
// every block reads all of them and comes to the same conclusion by itself.  With one block per row one SM pulled the
// row from L2 five times: at 151,936 elements 86 us by nucleus, 38 with a temperature alone, 6.5 greedy; now 28.5 / 13.0 / 3.4
// for one row, 37 / 19.5 / 4.3 for 19, 54 / 28 / 5.7 for 64 (from 75 rows on there is one block per row as before: 84 / 39 / 6.7).
// The threshold t is found ten bits a pass: a histogram, over the next ten bits of
// the patterns of e (positive floats order like their patterns), of the mass in each
// bin, as exact integers so that the order of the additions does not matter, then a
// scan from the top for the bin in which the mass crosses.  Three passes fix all
// thirty bits in which floats of (0, 1] can differ.  (A search of the pattern bit by
// bit, one pass a bit, took 1.1 ms a row at a vocabulary of 151,936.)
// The same logits and u give the same token on every run.
#include "common.cuh"
#include <cooperative_groups.h>
#include <limits.h>

namespace cg = cooperative_groups;

#define SAMPLE_THREADS 1024
#define SAMPLE_WARPS (SAMPLE_THREADS / 32)
#define SAMPLE_BINS 1024
#define SAMPLE_GROUPS 256  // groups of 32 elements per stretch: rows of up to 2^18 elements
static_assert(SAMPLE_BINS == SAMPLE_THREADS, "the scan below gives every thread one bin");

__device__ __forceinline__ float sample_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// f(index, value) for elements [i0, i1) of the row, each thread its share in ascending index order (i0 a multiple of 4).
// Sixteen elements a thread are asked for before the first is used (four 16-byte loads when the row allows it).
template <typename F>
__device__ __forceinline__ void row_for_each(const float* __restrict__ x, int i0, int i1, F f) {
    const int tid = threadIdx.x;
    if ((((uintptr_t)x) & 15) == 0) {
        const int n4 = i1 >> 2;
        const float4* x4 = reinterpret_cast<const float4*>(x);
        for (int j0 = (i0 >> 2) + tid; j0 < n4; j0 += SAMPLE_THREADS * 4) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * SAMPLE_THREADS;
                if (j < n4) v[u] = x4[j];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * SAMPLE_THREADS;
                if (j < n4) {
                    f(4 * j, v[u].x);
                    f(4 * j + 1, v[u].y);
                    f(4 * j + 2, v[u].z);
                    f(4 * j + 3, v[u].w);
                }
            }
        }
        for (int i = max(n4 << 2, i0) + tid; i < i1; i += SAMPLE_THREADS) f(i, x[i]);
    } else {
        for (int j0 = i0 + tid; j0 < i1; j0 += SAMPLE_THREADS * 4) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = j0 + u * SAMPLE_THREADS;
                if (i < i1) v[u] = x[i];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = j0 + u * SAMPLE_THREADS;
                if (i < i1) f(i, v[u]);
            }
        }
    }
}

// the lanes' values added up in lane order: lane l gets v_0 + ... + v_l
__device__ __forceinline__ float warp_scan(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += up;
    }
    return v;
}

__device__ __forceinline__ void block_argmax(float& v, int& idx, float* sv, int* si) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    __syncthreads();
    if (lane == 0) { sv[warp] = v; si[warp] = idx; }
    __syncthreads();
    v = lane < SAMPLE_WARPS ? sv[lane] : -INFINITY;
    idx = lane < SAMPLE_WARPS ? si[lane] : INT_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
}

__device__ __forceinline__ int block_min_int(int v, int* si) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) si[warp] = v;
    __syncthreads();
    v = lane < SAMPLE_WARPS ? si[lane] : INT_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// BLOCKS: blocks of a row's cluster, each with 32 / BLOCKS stretches that are dealt to as many warps as there are blocks.
// KEPT: the block keeps its part of the row in shared memory; otherwise later passes read it from memory again.
template <int BLOCKS, typename T>
__device__ __forceinline__ T* sample_at(cg::cluster_group& cluster, T* p, int block) {
    return BLOCKS > 1 ? cluster.map_shared_rank(p, block) : p;
}

template <int BLOCKS, bool KEPT>
__device__ __forceinline__ void sample_row(const float* __restrict__ logits, int ld, int V, const float* __restrict__ temperature,
                                           const float* __restrict__ top_p, const float* __restrict__ uniform, int* __restrict__ out) {
    cg::cluster_group cluster = cg::this_cluster();
    if (BLOCKS > 1) cluster.barrier_arrive();   // (here this block's shared memory exists: waited for before the first store into another's)
    pdl_wait();
    pdl_trigger();
    constexpr int STRETCHES = SAMPLE_WARPS / BLOCKS, BUFFERS = BLOCKS > 1 ? 2 : 1;
    extern __shared__ float slice_s[];
    __shared__ float sv[32];
    __shared__ int si[32];
    __shared__ unsigned hist_lo[BUFFERS][SAMPLE_BINS], hist_hi[BUFFERS][SAMPLE_BINS];
    __shared__ unsigned long long warp_total[SAMPLE_WARPS];
    __shared__ unsigned long long above_s;
    __shared__ int first_s;
    __shared__ float stretch_mass[STRETCHES];
    __shared__ float group_mass[STRETCHES][SAMPLE_GROUPS];
    __shared__ float best_of[BLOCKS];
    __shared__ int best_i_of[BLOCKS], cand_of[BLOCKS], last_of[BLOCKS];
    // (a row of one block: plain barriers, its own shared memory)
    auto sync = [&]() { if (BLOCKS > 1) cluster.sync(); else __syncthreads(); };
    const int rank = BLOCKS > 1 ? (int)cluster.block_rank() : 0;
    const int r = blockIdx.x / BLOCKS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* x = logits + (size_t)r * ld;
    // The row is cut into 32 stretches of `groups` groups of 32 elements; a block has 32 / BLOCKS of them.
    const int groups = ((V + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) >> 5;   // at most SAMPLE_GROUPS
    const int b0 = min(rank * STRETCHES * groups * 32, V), b1 = min((rank + 1) * STRETCHES * groups * 32, V);

    const float temp = temperature ? temperature[r] : 0.f;
    const bool greedy = !(temp > 1e-7f);
    float best = -INFINITY;
    int best_i = INT_MAX;
    row_for_each(x, b0, b1, [&](int i, float v) {
        if (v > best) { best = v; best_i = i; }  // ascending i: the first maximum stays
        if (KEPT && !greedy) slice_s[i - b0] = v;
    });
    const float* slice = KEPT ? slice_s : x + b0;   // the block's part of the row
    block_argmax(best, best_i, sv, si);
    if (BLOCKS > 1) {
        cluster.barrier_wait();   // every block of the cluster has started: another's shared memory may be written
        if (tid < BLOCKS) {   // every block gets every block's
            sample_at<BLOCKS>(cluster, best_of, tid)[rank] = best;
            sample_at<BLOCKS>(cluster, best_i_of, tid)[rank] = best_i;
        }
        sync();
        best = best_of[0];
        best_i = best_i_of[0];
#pragma unroll
        for (int b = 1; b < BLOCKS; ++b)   // (ascending index order)
            if (best_of[b] > best || (best_of[b] == best && best_i_of[b] < best_i)) { best = best_of[b]; best_i = best_i_of[b]; }
    }
    if (greedy) {   // (nobody reaches into another block's shared memory any more)
        if (rank == 0 && tid == 0) out[r] = best_i;
        return;
    }
    const float k = 1.4426950408889634f / temp;  // e_i = 2^((x_i - max) k)
    const float xmax = best;

    float threshold = 0.f;
    const float P = top_p ? top_p[r] : 1.f;
    if (P > 0.f && P < 1.f) {
        unsigned prefix = 0u;             // the bits of the threshold's pattern found so far
        unsigned long long above = 0ull;  // mass of the patterns above the bins still in question
        unsigned long long target = 0ull;
        int buf = 0;
        for (int shift = 20; shift >= 0; shift -= 10, buf ^= BUFFERS - 1) {
            // (a histogram is cleared two passes after it was read; the cluster barrier in between orders the two)
            hist_lo[buf][tid] = 0u;
            hist_hi[buf][tid] = 0u;
            if (tid == 0) first_s = SAMPLE_THREADS;
            __syncthreads();
            // All elements of a bin have the same exponent, so a bin's mass is the sum of
            // their 24-bit mantissas times a power of two; the mantissas' low and high 12
            // bits are summed apart, each sum below 2^30 (64-bit atomics in shared memory
            // are a compare-and-swap loop).
            auto count = [&](int, float v) {
                const unsigned pat = __float_as_uint(sample_ex2((v - xmax) * k));
                if (pat != 0u && (pat >> (shift + 10)) == prefix) {
                    const unsigned bin = (pat >> shift) & (SAMPLE_BINS - 1);
                    const unsigned m = (pat & 0x7FFFFFu) | 0x800000u;
                    atomicAdd(&hist_lo[buf][bin], m & 0xFFFu);
                    atomicAdd(&hist_hi[buf][bin], m >> 12);
                }
            };
            if (KEPT) {
                for (int i = tid; i < b1 - b0; i += SAMPLE_THREADS) count(i, slice[i]);
            } else {
                row_for_each(x, b0, b1, count);
            }
            sync();
            // thread t looks at bin 1023 - t: its mass in fixed point (2^40 for 1.0) ...
            const unsigned bin_of_thread = SAMPLE_BINS - 1 - tid;
            const int exponent = (int)(((((prefix << 10) | bin_of_thread) << shift) >> 23) & 0xFFu);
            unsigned lo = 0u, hi = 0u;
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                lo += sample_at<BLOCKS>(cluster, hist_lo[buf], b)[bin_of_thread];
                hi += sample_at<BLOCKS>(cluster, hist_hi[buf], b)[bin_of_thread];
            }
            unsigned long long s = ((unsigned long long)hi << 12) + lo;
            s = exponent >= 110 ? s << (exponent - 110) : (110 - exponent < 64 ? s >> (110 - exponent) : 0ull);
            // ... and with it the mass of all bins above it
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long up = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += up;
            }
            if (lane == 31) warp_total[warp] = s;
            __syncthreads();
            for (int w = 0; w < warp; ++w) s += warp_total[w];
            if (shift == 20) {  // the first pass has seen the whole row: the nucleus' target
                if (tid == SAMPLE_THREADS - 1) above_s = s;
                __syncthreads();
                target = (unsigned long long)((double)P * (double)above_s);
                __syncthreads();
            }
            // the highest bin with which the mass reaches the target
            if (above + s >= target) atomicMin(&first_s, tid);
            __syncthreads();
            // (if rounding left the target above everything, the lowest bin: everything is kept)
            const int chosen = first_s < SAMPLE_THREADS ? first_s : SAMPLE_THREADS - 1;
            if (tid == max(chosen - 1, 0)) above_s = chosen == 0 ? above : above + s;
            __syncthreads();
            above = above_s;
            prefix = (prefix << 10) | (unsigned)(SAMPLE_BINS - 1 - chosen);
            __syncthreads();
        }
        threshold = __uint_as_float(prefix);
    }

    // Kept mass, then the token.  The stretches of the row follow each other in index order; a stretch is walked in groups of
    // 32 consecutive elements, one a lane, and the kept mass of every group is noted, so that the walk for the token only
    // has to look at the groups' masses and then at one group.
    const int mine_s = warp / BLOCKS;   // the warp's stretch of the block's
    const int w0 = mine_s * groups * 32;       // (counted from b0)
    float* gm = group_mass[mine_s];
    int last_kept = -1;
    __syncthreads();   // (the slice is whole)
    for (int g0 = warp % BLOCKS; g0 < groups; g0 += 4 * BLOCKS) {
        float xv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int g = g0 + u * BLOCKS, i = w0 + g * 32 + lane;
            xv[u] = g < groups && b0 + i < b1 ? slice[i] : -INFINITY;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int g = g0 + u * BLOCKS;
            if (g >= groups) break;
            float e = sample_ex2((xv[u] - xmax) * k);   // (nothing there: 2^-inf = 0)
            if (!(e >= threshold) || xv[u] == -INFINITY) e = 0.f;
            const unsigned kept = __ballot_sync(0xffffffffu, e > 0.f);
            if (kept) last_kept = b0 + w0 + g * 32 + 31 - __clz(kept);
            const float incl = warp_scan(e, lane);
            if (lane == 31) gm[g] = incl;
        }
    }
    // (with several blocks the last kept element goes to the first with the rest, below; the barriers make the masses visible)
    const int my_last = last_kept >= 0 ? -last_kept : INT_MAX;
    const int last_neg = BLOCKS > 1 ? block_min_int(my_last, si) : 0;
    if (BLOCKS == 1) __syncwarp();   // (a stretch is its warp's)
    const bool leads = warp % BLOCKS == 0;   // one warp of every stretch goes on
    float mine = 0.f;   // the groups' masses added up in group order
    if (leads) {
        for (int c = 0; c < groups; c += 32) mine += __shfl_sync(0xffffffffu, warp_scan(c + lane < groups ? gm[c + lane] : 0.f, lane), 31);
        if (lane == 0) stretch_mass[mine_s] = mine;
    }
    sync();
    float excl = 0.f, total = 0.f;
    const int stretch = rank * STRETCHES + mine_s;
    for (int w = 0; w < SAMPLE_WARPS; ++w) {  // in index order, the same in every thread
        if (w == stretch) excl = total;
        total += sample_at<BLOCKS>(cluster, stretch_mass, w / STRETCHES)[w % STRETCHES];
    }
    const float target = uniform[r] * total;

    int cand = INT_MAX;
    if (leads && excl + mine > target) {
        // the token lies in this stretch or before it: the first group whose mass crosses ...
        float run = excl;
        int group = -1;
        for (int c = 0; c < groups && group < 0; c += 32) {
            const float incl = warp_scan(c + lane < groups ? gm[c + lane] : 0.f, lane);
            const unsigned hit = __ballot_sync(0xffffffffu, run + incl > target);
            if (hit) {
                const int l = __ffs(hit) - 1;
                group = c + l;
                const float before = __shfl_sync(0xffffffffu, incl, l > 0 ? l - 1 : 0);
                if (l > 0) run += before;
            } else {
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        if (group >= 0) {
            // ... and in it the first kept element with which the mass crosses
            const int i = w0 + group * 32 + lane;
            float e = 0.f;
            if (b0 + i < b1) {
                e = sample_ex2((slice[i] - xmax) * k);
                if (!(e >= threshold)) e = 0.f;
            }
            const float incl = warp_scan(e, lane);
            const unsigned hit = __ballot_sync(0xffffffffu, e > 0.f && run + incl > target);
            if (hit) cand = b0 + w0 + group * 32 + __ffs(hit) - 1;
        }
    }
    cand = block_min_int(cand, si);
    if (BLOCKS == 1) {
        if (cand == INT_MAX) {   // (uniform) rounding left nobody above the target: the last kept token
            const int neg = block_min_int(my_last, si);
            cand = neg == INT_MAX ? best_i : -neg;
        }
        if (tid == 0) out[r] = cand;
        return;
    }
    if (tid == 0) {
        sample_at<BLOCKS>(cluster, cand_of, 0)[rank] = cand;
        sample_at<BLOCKS>(cluster, last_of, 0)[rank] = last_neg;
    }
    sync();
    if (rank != 0 || tid != 0) return;
    int neg = last_of[0];
    cand = cand_of[0];
    for (int b = 1; b < BLOCKS; ++b) {
        cand = min(cand, cand_of[b]);
        neg = min(neg, last_of[b]);
    }
    out[r] = cand != INT_MAX ? cand : (neg == INT_MAX ? best_i : -neg);
}

template <int BLOCKS, bool KEPT>
__global__ void __cluster_dims__(BLOCKS, 1, 1) __launch_bounds__(SAMPLE_THREADS)
sample_cluster_kernel(const float* __restrict__ logits, int ld, int V, const float* __restrict__ temperature,
                      const float* __restrict__ top_p, const float* __restrict__ uniform, int* __restrict__ out) {
    sample_row<BLOCKS, KEPT>(logits, ld, V, temperature, top_p, uniform, out);
}
template <bool KEPT>
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int ld, int V, const float* __restrict__ temperature,
              const float* __restrict__ top_p, const float* __restrict__ uniform, int* __restrict__ out) {
    sample_row<1, KEPT>(logits, ld, V, temperature, top_p, uniform, out);
}

#define SAMPLE_PART_MAX (160 * 1024)   // most bytes of a row that a block keeps
#define SAMPLE_PART_MIN 12288          // fewest elements worth a block: below, the cluster's barriers cost more than the pass (301 elements: 9.8 us in one block, 18 in eight)
// All forms at the first call on a device: a later call may come from inside a stream capture.  `at_once`: how many clusters of
// 2, 4 and 8 blocks (a block fills an SM) find room together, which is less than the SMs divided by their blocks, as a cluster lies within one
// of the GPU's groups of SMs: 74, 33 and 15 on a B200.  (Chosen by the number of SMs, 37 rows of 151,936 by clusters of four, greedy, took 8.4 us;
// one block a row 6.5, clusters of two 5.2.)
struct SampleSetup {
    bool done;
    int at_once[3];
};
template <int BLOCKS>
static cudaError_t configure_sample_clusters(int* at_once) {
    cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel<BLOCKS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_PART_MAX);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(BLOCKS);
    cfg.blockDim = dim3(SAMPLE_THREADS);
    cfg.dynamicSmemBytes = SAMPLE_PART_MAX;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = BLOCKS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(at_once, sample_cluster_kernel<BLOCKS, true>, &cfg) != cudaSuccess) {
        *at_once = 0;   // (not to be had: no clusters of this size)
        cudaGetLastError();
    }
    return cudaSuccess;
}
static int configure_sample(const int** at_once) {
    static SampleSetup setups[VX_MAX_DEVICES];
    const int dev = vx_current_device();
    if (dev < 0) return VX_ERR_LIMIT;
    SampleSetup& setup = setups[dev];
    *at_once = setup.at_once;
    if (setup.done) return VX_OK;
    cudaError_t e = cudaFuncSetAttribute(sample_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_PART_MAX);
    if (e == cudaSuccess) e = configure_sample_clusters<2>(&setup.at_once[0]);
    if (e == cudaSuccess) e = configure_sample_clusters<4>(&setup.at_once[1]);
    if (e == cudaSuccess) e = configure_sample_clusters<8>(&setup.at_once[2]);
    if (e != cudaSuccess) return (int)e;
    setup.done = true;
    return VX_OK;
}

extern "C" int vx_sample(const float* logits, int ld, int rows, int vocab, const float* temperature,
                         const float* top_p, const float* uniform, int* out, cudaStream_t stream) {
    if (rows <= 0) return VX_OK;
    if (vocab <= 0 || ld < vocab) return VX_ERR_SHAPE;
    if (vocab > (1 << 18)) return VX_ERR_LIMIT;  // the fixed-point mass of a row has to fit 64 bits
    if (temperature && !uniform) return VX_ERR_SHAPE;
    const int* at_once;
    if (const int rc = configure_sample(&at_once)) return rc;
    // As many blocks a row as let all clusters run at once (a second round of clusters costs more than their blocks save),
    // and the row's parts in shared memory where they fit.
    int blocks = rows <= at_once[2] ? 8 : rows <= at_once[1] ? 4 : rows <= at_once[0] ? 2 : 1;
    while (blocks > 1 && vocab / blocks < SAMPLE_PART_MIN) blocks /= 2;
    const size_t groups = ((vocab + SAMPLE_WARPS - 1) / SAMPLE_WARPS + 31) >> 5;   // (as in the kernel)
    const size_t part = SAMPLE_WARPS / blocks * groups * 32 * sizeof(float);
    // A block keeps its part of the row where that fits and the row is read again; a row of one block only if it is short
    // (25,000 elements, 75 rows, us, kept and not: temperature 11.2 and 10.6, nucleus 22.0 and 21.5; 5,000: 5.8 and 5.9, 11.6 and 12.1).
    const bool kept = temperature && part <= SAMPLE_PART_MAX && (blocks > 1 || vocab <= SAMPLE_PART_MIN);
#define SAMPLE_GO(KERNEL, KEPT)                                                                                       \
    VX_LAUNCH_K(VX_K_SAMPLE, (KERNEL), rows * blocks, SAMPLE_THREADS, KEPT ? part : 0, stream, logits, ld, vocab, \
                temperature, top_p, uniform, out)
#define SAMPLE_CLUSTER(BLOCKS, KEPT) SAMPLE_GO((sample_cluster_kernel<BLOCKS, KEPT>), KEPT)
    if (kept) {
        if (blocks == 8) SAMPLE_CLUSTER(8, true);
        else if (blocks == 4) SAMPLE_CLUSTER(4, true);
        else if (blocks == 2) SAMPLE_CLUSTER(2, true);
        else SAMPLE_GO(sample_kernel<true>, true);
    } else {
        if (blocks == 8) SAMPLE_CLUSTER(8, false);
        else if (blocks == 4) SAMPLE_CLUSTER(4, false);
        else if (blocks == 2) SAMPLE_CLUSTER(2, false);
        else SAMPLE_GO(sample_kernel<false>, false);
    }
#undef SAMPLE_CLUSTER
#undef SAMPLE_GO
    VX_LAUNCH_CHECK();
    return VX_OK;
}
