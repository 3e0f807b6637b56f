// Paged causal attention, the general kernel: any head size up to 256 (values may
// have another size than keys), any number of heads and groups, any page size, an
// optional window with optionally kept first positions, an optional bias by distance,
// element type float or bfloat16.  It serves prompt portions and decoded
// tokens alike, and it is the whole of the 32-bit path.
//
// One block per (token, query head), or, in the 32-bit path of layers without a window or runs, per eight tokens and two
// heads (below).  The token's absolute position p gives its
// keys: j in [start, p], start = max(0, p + 1 - window) with a window, else 0; with
// keep_first > 0 also j in [0, min(keep_first, start)), at their true positions.  With
// chunk > 0 start is no less than p - p mod chunk: a token sees its own run of `chunk`
// positions only, the runs counted from the request's position 0.
// Key j of the token's request lies in page block_table[seq, j / S] at offset
// j % S; pools are [page, Hk, S, D] and [page, Hk, S, Dv]; query head h reads kv head
// h / (H / Hk).  score = q.k * scale - slope_h * (p - j) with
// slope_h = 2^(-bias_exp * (h + 1) / H), or no bias for bias_exp = 0.
// With `sinks` (a float32 per query head) the softmax's denominator also holds
// exp(sinks[h]): an entry without a key or a value, not scaled.  With gate_col >= 0
// head h's output is multiplied by sigmoid(g), g the element at column gate_col + h
// of the token's row of `q`.  With softcap c > 0 a scaled score s becomes c tanh(s / c) before
// anything else is done to it.  A value row starts every v_stride elements (Dv unless the caller
// says otherwise: a pool whose rows hold the value as the first Dv elements of the key, v_pool =
// k_pool and v_stride = D, is read as it lies).
//
// Each warp takes chunks of 32 keys (chunk c goes to warp c mod 4): it forms the dot products
// q.k in float32, one key per lane in the end, keeps a
// running maximum m, sum l and accumulator acc (online softmax), and adds the
// 32 values in key order.  The four warps' (m, l, acc) are merged in warp
// order.  The order of every addition depends only on the token's own key
// range, never on the batch around it, so a position's output is bit-identical
// however the tokens were cut into steps.
#include "common.cuh"

#define ATT_WARPS 4
#define ATT_MAX_D 256

// Four neighbouring elements with one load (16 bytes of float32, 8 of bfloat16).
__device__ __forceinline__ float4 att_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 att_load4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(u.x));
    const float2 b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// PARTS > 0: the sizes of keys and values, the stride of a value row and the pools' addresses are multiples of four elements.  What
// bounds this kernel is the latency of its loads and how many blocks are there to hide it: eight lanes fetch a key, four keys at a time
// (PARTS times 32 elements), and a value row comes as four neighbouring channels a lane.  Heads up to 128: one such batch of keys and
// four values ahead, in 64 registers, eight blocks an SM; larger heads two and four, four blocks.  (Four batches and sixteen values in 124 registers
// were slower wherever blocks are many.  us, a lane a key, which touches 32 rows with every load, that, and so: one float32 token on 400
// keys, 16 heads of 128, 42, 25, 22; 64 of them 125, 110, 52; 1,000 tokens in a window of 1,024 2490, 1334, 1158; bfloat16, 1,000 tokens,
// heads of 80 640, 905, 572, of 256 1258, 976, 557; 64 decoded on 600 keys, heads of 192, 136, 196, 83.  Slower than a lane a key: bfloat16 heads of 36,
// 1,000 tokens, 485, 510.)  PARTS 0: any sizes, a lane a key.
// Which form runs follows from the layer's sizes, so a position's sums have one order.
template <typename T, int PARTS>
__global__ void __launch_bounds__(ATT_WARPS * 32, PARTS == 0 ? 9 : (PARTS <= 4 ? 8 : 4)) paged_attention_generic_kernel(
    const T* __restrict__ q, int q_row_stride, const T* __restrict__ k_pool,
    const T* __restrict__ v_pool, const int* __restrict__ block_table, int max_blocks,
    const int* __restrict__ seq_of_token, const int* __restrict__ positions, T* __restrict__ out,
    int out_row_stride, float scale, int window, int H, int Hk, int D, int S, int Dv, int keep_first,
    float bias_exp, const float* __restrict__ sinks, int gate_col, float softcap, int v_stride, int v_share, int out_f32,
    int chunk) {
    pdl_wait();
    pdl_trigger();
    constexpr bool FOUR = PARTS > 0, SMALL = FOUR && PARTS <= 4;   // (SMALL: values up to 128 as well)
    __shared__ __align__(FOUR ? 16 : 4) float q_s[ATT_MAX_D];   // (aligned for the other form, its loop over d is half as fast)
    __shared__ float acc_s[ATT_WARPS][ATT_MAX_D];
    __shared__ float m_s[ATT_WARPS], l_s[ATT_WARPS];

    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hk = h / (H / Hk);
    const int seq = seq_of_token[t];
    const int kv_len = positions[t] + 1;
    int start = (window > 0 && kv_len > window) ? kv_len - window : 0;
    if (chunk > 0) start = max(start, kv_len - 1 - (kv_len - 1) % chunk);
    const int nkept = min(keep_first, start);   // kept first positions that lie before the window
    const float slope = bias_exp > 0.f ? exp2f(-bias_exp * (float)(h + 1) / (float)H) : 0.f;
    const int* bt = block_table + (size_t)seq * max_blocks;

    for (int d = threadIdx.x; d < (FOUR ? ATT_MAX_D : D); d += blockDim.x)
        q_s[d] = d < D ? to_f32(q[(size_t)t * q_row_stride + (size_t)h * D + d]) : 0.f;
    __syncthreads();

    constexpr int NR = SMALL ? 4 : ATT_MAX_D / 32;   // output channels of a lane
    float acc[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;

    const int nkeys = nkept + kv_len - start;   // the n-th visible key is j = n (kept) or start + n - nkept
    const int nchunks = (nkeys + 31) >> 5;
    for (int c = warp; c < nchunks; c += ATT_WARPS) {
        const int n = c * 32 + lane;
        const int j = n < nkept ? n : start + n - nkept;
        const bool valid = n < nkeys;
        size_t base = 0, kbase = 0;
        float s = -INFINITY;
        if (valid) {
            const int page = bt[j / S];
            base = ((size_t)page * Hk + hk) * S + (j % S);
            const T* kp = k_pool + base * D;
            kbase = base;
            if (v_share > 1) base = ((size_t)page * (Hk / v_share) + hk / v_share) * S + (j % S);
            if (!FOUR) {
                float dot = 0.f;
                for (int d = 0; d < D; ++d) dot += q_s[d] * to_f32(kp[d]);
                s = dot;
            }
        }
        const int nvalid = min(32, nkeys - c * 32);
        if (FOUR) {
            // eight lanes a key, four keys at a time: key 4 i + lane / 8 of the chunk
            constexpr int AHEAD = SMALL ? 1 : 2;
#pragma unroll 1
            for (int i0 = 0; i0 < 8; i0 += AHEAD) {
                float4 b[AHEAD][FOUR ? PARTS : 1];
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const int jj = 4 * (i0 + u) + (lane >> 3);
                    const T* kp = k_pool + (size_t)__shfl_sync(0xffffffffu, (unsigned long long)kbase, jj) * D + 4 * (lane & 7);
#pragma unroll
                    for (int r = 0; r < PARTS; ++r)
                        b[u][r] = jj < nvalid && 32 * r + 4 * (lane & 7) < D ? att_load4(kp + 32 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int r = 0; r < PARTS; ++r) {
                        const float4 a = *reinterpret_cast<const float4*>(q_s + 32 * r + 4 * (lane & 7));   // (zeros beyond D)
                        sum.x = fmaf(a.x, b[u][r].x, sum.x);
                        sum.y = fmaf(a.y, b[u][r].y, sum.y);
                        sum.z = fmaf(a.z, b[u][r].z, sum.z);
                        sum.w = fmaf(a.w, b[u][r].w, sum.w);
                    }
                    float dot = (sum.x + sum.y) + (sum.z + sum.w);
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                    dot = __shfl_sync(0xffffffffu, dot, 8 * (lane & 3));   // (lane's own key is 4 (lane / 4) + lane % 4)
                    if (i0 + u == lane >> 2) s = dot;
                }
            }
        }
        if (valid) {
            s *= scale;
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            s -= slope * (float)(kv_len - 1 - j);
        } else {
            s = -INFINITY;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.f;
        const float alpha = expf(m - m_new);  // m = -inf on the first chunk: 0
        l = l * alpha + warp_sum(p);
#pragma unroll
        for (int i = 0; i < NR; ++i) acc[i] *= alpha;
        if (FOUR) {
            constexpr int AHEAD = 4, VPARTS = SMALL ? 1 : 2;
#pragma unroll 1
            for (int j0 = 0; j0 < nvalid; j0 += AHEAD) {
                float4 v[AHEAD][VPARTS];
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const T* vp = v_pool + (size_t)__shfl_sync(0xffffffffu, (unsigned long long)base, j0 + u) * v_stride + lane * 4;
#pragma unroll
                    for (int r = 0; r < VPARTS; ++r)
                        v[u][r] = j0 + u < nvalid && lane * 4 + 128 * r < Dv ? att_load4(vp + 128 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const float pj = __shfl_sync(0xffffffffu, p, j0 + u);   // (0 beyond the last key)
#pragma unroll
                    for (int r = 0; r < VPARTS; ++r) {
                        acc[4 * r] = fmaf(pj, v[u][r].x, acc[4 * r]);
                        acc[4 * r + 1] = fmaf(pj, v[u][r].y, acc[4 * r + 1]);
                        acc[4 * r + 2] = fmaf(pj, v[u][r].z, acc[4 * r + 2]);
                        acc[4 * r + 3] = fmaf(pj, v[u][r].w, acc[4 * r + 3]);
                    }
                }
            }
        } else {
            for (int jj = 0; jj < nvalid; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, p, jj);
                const size_t bj = __shfl_sync(0xffffffffu, (unsigned long long)base, jj);
                const T* vp = v_pool + bj * v_stride;
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const int d = lane + 32 * i;
                    if (d < Dv) acc[i] += pj * to_f32(vp[d]);
                }
            }
        }
        m = m_new;
    }

    if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int d = FOUR ? lane * 4 + 128 * (i >> 2) + (i & 3) : lane + 32 * i;
        if (d < Dv) acc_s[warp][d] = acc[i];
    }
    __syncthreads();
    float M = -INFINITY;
    for (int w = 0; w < ATT_WARPS; ++w) M = fmaxf(M, m_s[w]);
    float L = 0.f;
    float wgt[ATT_WARPS];
    for (int w = 0; w < ATT_WARPS; ++w) {
        wgt[w] = (m_s[w] == -INFINITY) ? 0.f : expf(m_s[w] - M);
        L += l_s[w] * wgt[w];
    }
    if (sinks) {
        // the sink joins the denominator only; where it exceeds every score the reference moves to it
        const float sk = sinks[h];
        if (sk > M) {
            const float f = expf(M - sk);   // (M is finite: a token always sees itself)
            L = L * f + 1.f;
            for (int w = 0; w < ATT_WARPS; ++w) wgt[w] *= f;
        } else {
            L += expf(sk - M);
        }
    }
    float gate = 1.f;
    if (gate_col >= 0) gate = 1.f / (1.f + expf(-to_f32(q[(size_t)t * q_row_stride + gate_col + h])));
    for (int d = threadIdx.x; d < Dv; d += blockDim.x) {
        float o = 0.f;
        for (int w = 0; w < ATT_WARPS; ++w) o += acc_s[w][d] * wgt[w];
        if (out_f32) reinterpret_cast<float*>(out)[(size_t)t * out_row_stride + (size_t)h * Dv + d] = o / L * gate;
        else out[(size_t)t * out_row_stride + (size_t)h * Dv + d] = from_f32<T>(o / L * gate);
    }
}

// ---- the same for float32 layers in which every token sees all keys up to its own ----
// There the chunks of 32 keys lie alike for all tokens of a request, so a block takes up to eight of its neighbouring tokens
// (from a position that is a multiple of eight to the next) and up to two heads of a kv head, and brings every key and value
// into shared memory once for all of them: four chunks a round, sixteen warps: warp w works on chunk 4 round + w mod 4 for every fourth
// query (token and head) of the block, from w / 4 on.  The next round's keys come while this one's values are used, and the other way round.
// A token's chunks go to the same four running sums in the same order, and are merged alike, whatever tokens are in its block.
// What bounds it: a round's chain (loads, products, sums over eight lanes, softmax, values; about 5 us a round; with four queries a warp
// it spills 148 bytes at its 128 registers).  16 heads of 128, 8 kv heads, us, a
// block per token and head and this: 96 prompt tokens beside 3 on 200 to 400 keys 54, 23; 96 prompt tokens alone 26, 16; one token on 400 keys 42,
// 22; four on 800 79, 39; 150 prompt tokens 52, 35.
#define ATS_TOKENS 8
#define ATS_HEADS 2
#define ATS_QUERIES (ATS_TOKENS * ATS_HEADS)
#define ATS_KEYS 128     // keys of a round
#define ATS_DIM 128
#define ATS_THREADS 512
#define ATS_WARPS (ATS_THREADS / 32)
#define ATS_SMEM ((2 * ATS_KEYS * ATS_DIM + ATS_QUERIES * ATS_DIM + ATS_QUERIES * ATS_KEYS) * 4)

__device__ __forceinline__ void ats_copy(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

struct AtsCall {
    const float *q, *k_pool, *v_pool;
    const int *block_table, *seq_of_token, *positions;
    float* out;
    const float* sinks;
    float scale, bias_exp, softcap;
    int q_row_stride, max_blocks, out_row_stride, tokens, H, Hk, D, S, Dv, gate_col, v_stride, v_share;
};

// A block's rounds with MINE queries a warp at most: query 4 u + warp / 4 for u < MINE.
template <int MINE>
__device__ __forceinline__ void ats_rounds(const AtsCall& g, const int* __restrict__ bt, int pos0, int nt, int nh, int h0, int hk, float* k_s, float* v_s,
                                           const float* q_s, float* p_all, float (*m_s)[ATS_QUERIES], float (*l_s)[ATS_QUERIES]) {
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int slot = warp & 3, quarter = warp >> 2, nq = nt * nh, keys = pos0 + nt, D = g.D, S = g.S;
    float* p_s = p_all + warp * MINE * 32;   // [this warp's queries][keys of the chunk]
    float m[MINE], l[MINE], acc[MINE][4], slope[MINE];
    int last[MINE];   // the last key that a query sees (-1: there is no such query)
#pragma unroll
    for (int u = 0; u < MINE; ++u) {
        const int i = 4 * u + quarter;
        last[u] = i < nq ? pos0 + i / nh : -1;
        slope[u] = g.bias_exp > 0.f ? exp2f(-g.bias_exp * (float)(h0 + i % nh + 1) / (float)g.H) : 0.f;
        m[u] = -INFINITY;
        l[u] = acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.f;
    }
    // a warp brings eight keys of a round, its first eight lanes know where they lie
    struct Row { int page, offset; };
    auto row_of = [&](int base) {
        const int j = base + warp * 8 + (lane & 7);
        return j < keys ? Row{bt[j / S], j % S} : Row{0, 0};
    };
    auto fetch = [&](float* dst, const float* pool, int heads, int head, int dim, int stride, int base, const Row& row) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int page = __shfl_sync(0xffffffffu, row.page, r), offset = __shfl_sync(0xffffffffu, row.offset, r);
            if (base + warp * 8 + r < keys && lane * 4 < dim)
                ats_copy(dst + (warp * 8 + r) * ATS_DIM + lane * 4, pool + (((size_t)page * heads + head) * S + offset) * stride + lane * 4);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int vheads = g.Hk / g.v_share, vhead = hk / g.v_share;
    Row row = row_of(0);
    fetch(k_s, g.k_pool, g.Hk, hk, D, D, 0, row);
    fetch(v_s, g.v_pool, vheads, vhead, g.Dv, g.v_stride, 0, row);
    for (int base = 0; base < keys; base += ATS_KEYS) {
        const int next = base + ATS_KEYS;
        row = row_of(next);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");   // (the keys; the values are still on their way)
        __syncthreads();
        const int first = base + slot * 32;   // the chunk's first key
        const bool work = first < keys;
        bool whole = true;   // every query of the warp sees all of the chunk
        if (work) {
            const float* kc = k_s + slot * 32 * ATS_DIM;
            float4 a[MINE][4];
#pragma unroll
            for (int u = 0; u < MINE; ++u)
#pragma unroll
                for (int r = 0; r < 4; ++r) a[u][r] = *reinterpret_cast<const float4*>(q_s + (4 * u + quarter) * ATS_DIM + 32 * r + 4 * (lane & 7));
            float s[MINE];
            // eight lanes a key, four keys at a time: key 4 i + lane / 8 of the chunk
#pragma unroll 2
            for (int i = 0; i < 8; ++i) {
                float4 b[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int d = 32 * r + 4 * (lane & 7);
                    b[r] = d < D ? *reinterpret_cast<const float4*>(kc + (4 * i + (lane >> 3)) * ATS_DIM + d) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                float dot[MINE];
#pragma unroll
                for (int u = 0; u < MINE; ++u) {
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        sum.x = fmaf(a[u][r].x, b[r].x, sum.x);
                        sum.y = fmaf(a[u][r].y, b[r].y, sum.y);
                        sum.z = fmaf(a[u][r].z, b[r].z, sum.z);
                        sum.w = fmaf(a[u][r].w, b[r].w, sum.w);
                    }
                    dot[u] = (sum.x + sum.y) + (sum.z + sum.w);
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1)
#pragma unroll
                    for (int u = 0; u < MINE; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], o);
#pragma unroll
                for (int u = 0; u < MINE; ++u) {
                    const float mine = __shfl_sync(0xffffffffu, dot[u], 8 * (lane & 3));   // (lane's own key is 4 (lane / 4) + lane % 4)
                    if (i == lane >> 2) s[u] = mine;
                }
            }
            float x[MINE], mx[MINE], sum[MINE];
#pragma unroll
            for (int u = 0; u < MINE; ++u) {
                x[u] = s[u] * g.scale;
                if (g.softcap > 0.f) x[u] = g.softcap * tanhf(x[u] / g.softcap);
                x[u] -= slope[u] * (float)(last[u] - first - lane);
                if (first + lane > last[u]) x[u] = -INFINITY;
                mx[u] = x[u];
                whole = whole && (last[u] < 0 || first + 31 <= last[u]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < MINE; ++u) mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], o));
#pragma unroll
            for (int u = 0; u < MINE; ++u) {
                mx[u] = fmaxf(m[u], mx[u]);
                sum[u] = first + lane <= last[u] ? expf(x[u] - mx[u]) : 0.f;
                p_s[u * 32 + lane] = sum[u];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < MINE; ++u) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
#pragma unroll
            for (int u = 0; u < MINE; ++u) {
                if (first > last[u]) continue;   // (uniform: a chunk past the query's last key leaves its sums alone)
                const float alpha = expf(m[u] - mx[u]);   // m = -inf on the first chunk: 0
                l[u] = l[u] * alpha + sum[u];
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[u][e] *= alpha;
                m[u] = mx[u];
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();   // (the values are there, the keys have been used)
        if (next < keys) fetch(k_s, g.k_pool, g.Hk, hk, D, D, next, row);
        if (work) {
            const float* vc = v_s + slot * 32 * ATS_DIM;
            const int n = min(32, keys - first);
#pragma unroll 2
            for (int j0 = 0; j0 < n; j0 += 4) {
                float4 v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(vc + (j0 + e) * ATS_DIM + lane * 4);
#pragma unroll
                for (int u = 0; u < MINE; ++u) {
                    const float4 p4 = *reinterpret_cast<const float4*>(p_s + u * 32 + j0);
                    const float pj[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // (a value that a query does not see must not touch its sums, whatever it is)
                        if (!whole && first + j0 + e > last[u]) continue;
                        acc[u][0] = fmaf(pj[e], v[e].x, acc[u][0]);
                        acc[u][1] = fmaf(pj[e], v[e].y, acc[u][1]);
                        acc[u][2] = fmaf(pj[e], v[e].z, acc[u][2]);
                        acc[u][3] = fmaf(pj[e], v[e].w, acc[u][3]);
                    }
                }
            }
        }
        __syncthreads();
        if (next < keys) fetch(v_s, g.v_pool, vheads, vhead, g.Dv, g.v_stride, next, row);
    }
    float* acc_s = k_s;   // [slot][query][channel], in place of the keys
#pragma unroll
    for (int u = 0; u < MINE; ++u) {
        const int i = 4 * u + quarter;
        if (i >= nq) continue;
        if (lane == 0) { m_s[slot][i] = m[u]; l_s[slot][i] = l[u]; }
        *reinterpret_cast<float4*>(acc_s + (slot * ATS_QUERIES + i) * ATS_DIM + lane * 4) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(ATS_THREADS, 1) paged_attention_shared_kernel(const AtsCall g) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) float ats[];
    float *k_s = ats, *v_s = ats + ATS_KEYS * ATS_DIM, *q_s = v_s + ATS_KEYS * ATS_DIM, *p_s = q_s + ATS_QUERIES * ATS_DIM;
    __shared__ float m_s[4][ATS_QUERIES], l_s[4][ATS_QUERIES];
    __shared__ int count_s[ATS_WARPS], start_s;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int *seq_of_token = g.seq_of_token, *positions = g.positions;
    // (tokens at positions that do not follow each other make more runs than the grid has blocks: then a block takes several)
    for (int wanted = blockIdx.x;; wanted += gridDim.x) {
    // the block's tokens begin with the wanted-th that begins a run: at a multiple of eight, or after another request's
    if (threadIdx.x == 0) start_s = -1;
    for (int base = 0, seen = 0; base < g.tokens; base += ATS_THREADS) {
        const int t = base + threadIdx.x;
        const bool begins = t < g.tokens && (t == 0 || !(positions[t] & (ATS_TOKENS - 1)) || seq_of_token[t - 1] != seq_of_token[t] ||
                                             positions[t - 1] != positions[t] - 1);
        const unsigned votes = __ballot_sync(0xffffffffu, begins);
        __syncthreads();   // (start_s, and the counts of the pass before)
        if (lane == 0) count_s[warp] = __popc(votes);
        __syncthreads();
        int before = seen;
#pragma unroll
        for (int w = 0; w < ATS_WARPS; ++w) {
            before += w < warp ? count_s[w] : 0;
            seen += count_s[w];
        }
        if (begins && before + __popc(votes & ((1u << lane) - 1)) == wanted) start_s = t;
        if (seen > wanted) break;   // (uniform)
    }
    __syncthreads();
    const int t0 = start_s;
    if (t0 < 0) return;   // (uniform)
    const int seq = seq_of_token[t0], pos0 = positions[t0], H = g.H, Hk = g.Hk;
    int nt = 1;
    while (nt < ATS_TOKENS && t0 + nt < g.tokens && ((pos0 + nt) & (ATS_TOKENS - 1)) && seq_of_token[t0 + nt] == seq && positions[t0 + nt] == pos0 + nt) ++nt;
    const int group = H / Hk, per_kv = (group + ATS_HEADS - 1) / ATS_HEADS;
    const int hk = blockIdx.y / per_kv, h0 = hk * group + (blockIdx.y % per_kv) * ATS_HEADS, nh = min(ATS_HEADS, (hk + 1) * group - h0);
    const int nq = nt * nh;   // query i: token i / nh, head h0 + i % nh
    for (int e = threadIdx.x; e < ATS_QUERIES * ATS_DIM; e += ATS_THREADS) {
        const int i = e / ATS_DIM, d = e % ATS_DIM;
        q_s[e] = i < nq && d < g.D ? g.q[(size_t)(t0 + i / nh) * g.q_row_stride + (size_t)(h0 + i % nh) * g.D + d] : 0.f;
    }
    const int* bt = g.block_table + (size_t)seq * g.max_blocks;
    if (nq > 8) ats_rounds<4>(g, bt, pos0, nt, nh, h0, hk, k_s, v_s, q_s, p_s, m_s, l_s);
    else if (nq > 4) ats_rounds<2>(g, bt, pos0, nt, nh, h0, hk, k_s, v_s, q_s, p_s, m_s, l_s);
    else ats_rounds<1>(g, bt, pos0, nt, nh, h0, hk, k_s, v_s, q_s, p_s, m_s, l_s);
    const float* acc_s = k_s;
    for (int i = warp; i < nq; i += ATS_WARPS) {   // a warp merges a query's four sums
        const int t = t0 + i / nh, h = h0 + i % nh;
        float M = -INFINITY, L = 0.f, wgt[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) M = fmaxf(M, m_s[w][i]);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            wgt[w] = m_s[w][i] == -INFINITY ? 0.f : expf(m_s[w][i] - M);
            L += l_s[w][i] * wgt[w];
        }
        if (g.sinks) {
            const float sk = g.sinks[h];
            if (sk > M) {
                const float f = expf(M - sk);
                L = L * f + 1.f;
#pragma unroll
                for (int w = 0; w < 4; ++w) wgt[w] *= f;
            } else {
                L += expf(sk - M);
            }
        }
        float gate = 1.f;
        if (g.gate_col >= 0) gate = 1.f / (1.f + expf(-g.q[(size_t)t * g.q_row_stride + g.gate_col + h]));
        for (int d = lane; d < g.Dv; d += 32) {
            float o = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) o += acc_s[(w * ATS_QUERIES + i) * ATS_DIM + d] * wgt[w];
            g.out[(size_t)t * g.out_row_stride + (size_t)h * g.Dv + d] = o / L * gate;
        }
    }
    __syncthreads();
    }
}

// `v_share` > 1: that many consecutive key heads read one value head (the value pool has Hk / v_share heads);
// `out_f32`: the output is written as float32 whatever the element type of the inputs; `chunk` > 0: see
// the top (it does not go with kept first positions).
// `requests` (0: unknown): how many the tokens belong to, at most.
extern "C" int vx_paged_attention_generic_requests(const void* q, int q_row_stride, const void* k_pool,
                                                   const void* v_pool, const int* block_table, int max_blocks,
                                                   const int* seq_of_token, const int* positions, void* out,
                                                   int out_row_stride, float scale, int window, int tokens,
                                                   int H, int Hk, int D, int S, int dtype, int Dv, int keep_first,
                                                   float bias_exp, const float* sinks, int gate_col, float softcap,
                                                   int v_stride, int v_share, int out_f32, int chunk, int requests, cudaStream_t stream) {
    if (tokens <= 0) return VX_OK;
    if (Dv <= 0) Dv = D;
    if (v_stride <= 0) v_stride = Dv;
    if (v_share <= 0) v_share = 1;
    if (Hk % v_share) return VX_ERR_SHAPE;
    if (v_stride < Dv || softcap < 0.f) return VX_ERR_SHAPE;
    if (H <= 0 || Hk <= 0 || H % Hk || D <= 0 || D > ATT_MAX_D || Dv > ATT_MAX_D || S <= 0 || max_blocks <= 0)
        return VX_ERR_SHAPE;
    if (window < 0 || keep_first < 0 || bias_exp < 0.f || chunk < 0 || (chunk && keep_first)) return VX_ERR_SHAPE;
    dim3 grid(tokens, H);
    if (dtype != VX_F32 && dtype != VX_BF16) return VX_ERR_DTYPE;
    const bool four = !((D | Dv | v_stride) & 3) && !((((uintptr_t)k_pool) | ((uintptr_t)v_pool)) & (dtype == VX_F32 ? 15 : 7));
    const bool small = D <= 128 && Dv <= 128;
    // Tokens that share their keys and values: not where most requests bring a token of their own and the blocks, which fill an SM each, would take
    // turns (the form below has the same bits.  Decoded tokens, us, shared and not: 64 on 100 keys, 16 heads on 8, 33, 14; on 1,500 277, 160;
    // 16 heads on 16, 32 on 100 34, 9; on 400 95, 49; 8 heads on 2, 64 on 1,500 125, 130.  In one turn: 8 on 400 keys 24, 22; on 1,500 70, 117).
    static int sms_cache[VX_MAX_DEVICES];
    const int groups = Hk * ((H / Hk + ATS_HEADS - 1) / ATS_HEADS);
    const bool shared = requests <= 0 || tokens >= 4ll * requests || (long long)tokens * groups <= vx_sm_count(sms_cache);
    if (dtype == VX_F32 && four && small && window == 0 && chunk == 0 && shared) {
        static bool configured[VX_MAX_DEVICES];
        if (int rc = vx_configure_smem(paged_attention_shared_kernel, ATS_SMEM, configured)) return rc;
        // (runs of tokens: a request's neighbouring ones have one for every eight positions, and two that are not whole)
        const int runs = requests > 0 && requests < tokens ? (int)min((long long)tokens, tokens / ATS_TOKENS + 2ll * requests) : tokens;
        const AtsCall g = {(const float*)q, (const float*)k_pool, (const float*)v_pool, block_table, seq_of_token, positions, (float*)out, sinks, scale,
                           bias_exp, softcap, q_row_stride, max_blocks, out_row_stride, tokens, H, Hk, D, S, Dv, gate_col, v_stride, v_share};
        VX_LAUNCH_K(VX_K_ATTENTION, paged_attention_shared_kernel, dim3(runs, groups), ATS_THREADS, ATS_SMEM, stream, g);
        VX_LAUNCH_CHECK();
        return VX_OK;
    }
    const int parts = !four ? 0 : (!small ? 8 : (D <= 64 ? 2 : (D + 31) / 32));
#define ATT_GO(T, P_)                                                                                                                    \
    VX_LAUNCH_K(VX_K_ATTENTION, (paged_attention_generic_kernel<T, P_>), grid, ATT_WARPS * 32, 0, stream, (const T*)q, q_row_stride,     \
                (const T*)k_pool, (const T*)v_pool, block_table, max_blocks, seq_of_token, positions, (T*)out, out_row_stride, scale, \
                window, H, Hk, D, S, Dv, keep_first, bias_exp, sinks, gate_col, softcap, v_stride, v_share, out_f32, chunk)
#define ATT_OF(T)                          \
    do {                                   \
        if (parts == 0) ATT_GO(T, 0);      \
        else if (parts == 2) ATT_GO(T, 2); \
        else if (parts == 3) ATT_GO(T, 3); \
        else if (parts == 4) ATT_GO(T, 4); \
        else ATT_GO(T, 8);                 \
    } while (0)
    if (dtype == VX_F32) ATT_OF(float);
    else ATT_OF(bf16);
#undef ATT_OF
#undef ATT_GO
    VX_LAUNCH_CHECK();
    return VX_OK;
}
