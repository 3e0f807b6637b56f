// Paged attention for decoded tokens (one query per request), bfloat16, with the
// key/value range of a request split into pieces of fixed size that are worked on
// independently and joined by a second, small kernel.
//
// The unit of work is a PIECE: `piece_tiles` tiles of 16 keys of one kv head of one request and ALL the query heads of
// that kv head (the group), so every key and value is read from memory once.  A warp streams tiles through a cp.async
// ring of its own in shared memory (no barrier between warps), computes scores and outputs with mma.sync.m16n8k16
// (bf16 in, float32 out) and keeps maximum, sum and accumulator per query head in float32 (softmax, base 2).  A request
// whose whole range is one piece gets its output written at once; otherwise the unnormalised accumulator and (max, sum)
// go to scratch, and the join kernel (one block per request and head) adds the pieces.
//
// Piece boundaries depend only on the request's own key range (fixed number of
// keys per piece), never on the batch, so a request's output does not depend on
// what else is in the step.
//
// How the pieces are spread over blocks changes nothing in what is computed, so it is chosen per launch (microseconds of a
// layer with its join on a B200, 32 query and 8 kv heads of 128, one after another under programmatic launch):
//   - up to one piece per SM: a block of eight warps per piece, one sub-piece each (1 request of 500 keys: 5.6, a warp
//     per piece 8.2; 4,096 keys: 7.7 and 9.3; from two pieces per SM on the warp per piece is ahead, 10.3 and 13.2 at 8,192);
//   - more: a warp, as a block of its own, per piece, with room for two sub-pieces (32 KB at D = 128), four blocks an SM.
//     Small blocks leave the fewest SMs idle at the end (8 requests of 4,096 keys: 26.4; 20 of 2,000: 33; 64 of 4,096:
//     165, which is the copy bandwidth).
// The blocks an SM holds are set by the part of its L1 that the kernel asks for as shared memory (configure_decode): all of
// it would take a sixth block, and win at 20 requests of 2,000 keys (30), but an SM keeps the split as long as kernels
// follow each other without a gap, and the products after this one then read their rows through the 28 KB that is left:
// steps of 1 request of 16,000 keys and of 8 of 4,096 took 1,058 and 1,687 us instead of 983 and 1,447 (12 layers of the 4B, 8B
// shape), and 1,033 and 1,488 with three blocks an SM.
// Groups above eight heads of 128 take twice the instructions a key, and where the pieces are many a lone warp of a scheduler is the bound: 64
// requests of 1,000 keys, 64 heads on 4, 36 us, 64 of 4,096 105 (heads in the 16 rows, eight warps an SM: 32 and 100; but 16
// requests of 4,096 30.3 against 29.7 now, 64 of 300 20.1 against 18.0, one of 16,000 with 32 heads on 2 18.6 against 8.8).
// Before, blocks of 4 to 6 warps walked pieces tile by tile, each tile with a softmax of its own and the queries in
// the 16 rows of mma.sync: 15.2 us for one request of 500 keys (now 5.6), 20.5 for one of 16,000 (14.0), 41.5 for 20 of
// 2,000 (33), 173 for 64 of 4,096 (165).
//
// Launched programmatically (see common.cuh) a warp asks for its first tiles before it
// waits for the kernel before it, unless they reach the request's newest position: the
// only thing that kernel may write into the pools is the key and value at position
// kv_len - 1 of each request (which is what writing the step's new tokens does).
//
// Sizes: head size 64 or 128; page size a multiple of 16; group size up to 16;
// any number of heads; an optional window.  Other sizes are refused (the caller
// then uses the general kernel).
#include "common.cuh"
#include "mma_helpers.cuh"

#define LOG2E 1.4426950408889634f
#define DEC_CARVEOUT 57   // per cent of an SM's 228 KB: 132 KB, four rings or one block of eight warps at D = 128

// A piece is worked on in sub-pieces of DEC_SUB tiles (32 keys): each has a maximum, a sum and an accumulator of its
// own, and a piece's sub-pieces are folded together in order.  A warp that walks a whole piece folds as it goes; a
// block that gives every sub-piece a warp of its own folds through shared memory, with the same operations in the same
// order, so that both give the same bits.  (Sub-pieces of 64 keys: 5 % fewer instructions a key, but rings of 64 KB, three
// an SM: 17.2 instead of 14.1 us for one request of 16,000 keys, 32 instead of 30 for 20 of 2,000.)
//
// Scores and outputs are formed transposed, S^T = K Q^T and O^T = V^T P^T: keys (then channels) fill the 16-row side of
// mma.sync and the group's query heads the 8-column side (NG = 1 or 2 tiles of 8 heads).  The other way round a group of
// 2 or 4 heads leaves most of the 16 rows empty and needs twice the instructions and accumulator registers.  A lone warp
// is bound by the instructions it issues, about one in five cycles: a sub-piece is one softmax, its tiles' score chains
// are independent, and addresses are constants away from a few registers (DecLane).
#define DEC_SUB 2

// Maximum (base 2), sum and accumulator of a group's heads: a thread's heads are 8 n + (lane % 4) * 2 + {0, 1}, its
// channels 16 i + lane / 4 (+ 8).  The sum is this thread's share; the eight shares are added at the end.
template <int D, int NG>
struct DecPart {
    float o[D / 16][NG][4];
    float m[NG][2], l[NG][2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int n = 0; n < NG; ++n) {
#pragma unroll
            for (int i = 0; i < D / 16; ++i) o[i][n][0] = o[i][n][1] = o[i][n][2] = o[i][n][3] = 0.f;
            m[n][0] = m[n][1] = -INFINITY;
            l[n][0] = l[n][1] = 0.f;
        }
    }
};

// What folding (m, l, o) with (m2, l2, o2) multiplies each side with; -inf - (-inf) must not be formed.
__device__ __forceinline__ void fold_factors(float& m, float m2, float& a, float& b) {
    const float top = fmaxf(m, m2);
    a = m == -INFINITY ? 0.f : exp2f(m - top);
    b = m2 == -INFINITY ? 0.f : exp2f(m2 - top);
    m = top;
}
__device__ __forceinline__ float fold_add(float x, float a, float x2, float b) { return __fmaf_rn(x, a, __fmul_rn(x2, b)); }

__device__ __forceinline__ unsigned transpose_8x8(unsigned x) {
    unsigned y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}

// Where a lane writes and reads in a tile ([16 keys][D] bf16, 16-byte chunks of a row XOR-swizzled with the row index so
// that ldmatrix reads hit distinct banks).  All that differs between the instructions of a tile, and between tiles, is
// added as a constant: what bounds a warp here is how many instructions it issues a key.
template <int D>
struct DecLane {
    static constexpr int ROW = D * 2, PER_ROW = D / 8, ROWS = 32 / PER_ROW;   // (rows a copy instruction of the warp covers)
    unsigned put[4], k[4], v[4];
    __device__ __forceinline__ explicit DecLane(int lane) {
        const int mi = lane >> 3, kr = ((mi & 1) << 3) + (lane & 7), vr = ((mi >> 1) << 3) + (lane & 7);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = lane / PER_ROW + ROWS * i;
            put[i] = r * ROW + (((lane % PER_ROW) ^ (r & 7)) << 4);
            k[i] = kr * ROW + (((2 * i + (mi >> 1)) ^ (kr & 7)) << 4);
            v[i] = vr * ROW + (((2 * i + (mi & 1)) ^ (vr & 7)) << 4);
        }
    }
    // copy i of a tile; the A operand of score step i; the A operand of channels 16 i
    __device__ __forceinline__ unsigned put_at(int i) const { return put[i & 3] + (i >> 2) * 4 * ROWS * ROW; }
    __device__ __forceinline__ unsigned k_at(int i) const { return k[i & 3] + (i >> 2) * 128; }
    __device__ __forceinline__ unsigned v_at(int i) const { return v[i & 3] + (i >> 2) * 128; }
};
__device__ __forceinline__ void cp_async16_at(unsigned smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem));
}
__device__ __forceinline__ void ldmatrix_x4_at(unsigned (&r)[4], unsigned smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem));
}
__device__ __forceinline__ void ldmatrix_x4_trans_at(unsigned (&r)[4], unsigned smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem));
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// Which 16 rows of the pools tile `tile` of kv head hk is (rows counted in sixteens: 2^31 of them are 8 TB at D = 128).
__device__ __forceinline__ int dec_tile_rows(const int* __restrict__ bt, int tile, int hk, int Hk, int S) {
    const int per_page = S >> 4;
    return (bt[tile / per_page] * Hk + hk) * per_page + tile % per_page;
}
// Asks for a tile: keys, then values.
template <int D>
__device__ __forceinline__ void dec_ask_tile(unsigned smem, const bf16* __restrict__ k_lane, const bf16* __restrict__ v_lane, int rows,
                                             const DecLane<D>& at) {
    const bf16* kg = k_lane + (size_t)rows * (16 * D);
    const bf16* vg = v_lane + (size_t)rows * (16 * D);
#pragma unroll
    for (int i = 0; i < D / 16; ++i) cp_async16_at(smem + at.put_at(i), kg + i * 256);
#pragma unroll
    for (int i = 0; i < D / 16; ++i) cp_async16_at(smem + 16 * D * 2 + at.put_at(i), vg + i * 256);
}

// The queries of kv head hk's group: the B operand, kept in registers.
template <int D, int NG>
__device__ __forceinline__ void dec_load_queries(unsigned (&qf)[D / 16][NG][2], const bf16* __restrict__ q, int G, int lane) {
#pragma unroll
    for (int n = 0; n < NG; ++n) {
        const int g = 8 * n + (lane >> 2);
        const bf16* row = q + (size_t)g * D + (lane & 3) * 2;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            qf[kk][n][0] = g < G ? *reinterpret_cast<const unsigned*>(row + kk * 16) : 0u;
            qf[kk][n][1] = g < G ? *reinterpret_cast<const unsigned*>(row + kk * 16 + 8) : 0u;
        }
    }
}

// A sub-piece: `tiles` (1 to DEC_SUB) tiles in shared memory, one behind the other from `smem`, first key key0.
// `done(t)` is called (by the whole warp) when tile t's place is free.
template <int D, int NG, typename Done>
__device__ __forceinline__ void dec_sub_piece(DecPart<D, NG>& part, const unsigned (&qf)[D / 16][NG][2], unsigned smem,
                                              const DecLane<D>& at, int tiles, int key0, int start, int kv_len, float scale_log2,
                                              int lane, Done done) {
    constexpr int TILE = 16 * D * 2;
    if (key0 + (tiles << 4) > kv_len) {
        // Rows past the last key were never written (they may hold anything,
        // NaN included): their probabilities are zero, but 0 * NaN is NaN in
        // the tensor core, so the value rows are cleared.
        const unsigned vs = smem + (tiles - 1) * 2 * TILE + TILE;
        for (int c = lane; c < 16 * (D / 8); c += 32)
            if (key0 + ((tiles - 1) << 4) + c / (D / 8) >= kv_len)
                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(vs + c * 16), "r"(0) : "memory");
        __syncwarp();
    }
    float s[DEC_SUB][NG][4];
#pragma unroll
    for (int t = 0; t < DEC_SUB; ++t)
#pragma unroll
        for (int n = 0; n < NG; ++n) s[t][n][0] = s[t][n][1] = s[t][n][2] = s[t][n][3] = 0.f;
    const bool whole = tiles == DEC_SUB;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
        for (int t = 0; t < DEC_SUB; ++t) {
            if (t > 0 && !whole && t >= tiles) continue;
            unsigned a[4];
            ldmatrix_x4_at(a, smem + t * 2 * TILE + at.k_at(kk));
#pragma unroll
            for (int n = 0; n < NG; ++n) mma_bf16(s[t][n], a, qf[kk][n][0], qf[kk][n][1]);
        }
    // scale, mask, softmax over the sub-piece's keys (base 2); keys from key_end on are past the last, or another piece's (a piece
    // of an odd number of tiles ends with a sub-piece of one)
    const int key_end = min(kv_len, key0 + (tiles << 4));
    const bool inside = key0 >= start && key0 + 16 * DEC_SUB <= key_end;
    unsigned p[DEC_SUB][NG][2];   // [keys lane/4 .. | + 8], two heads each, then transposed: two keys of one head
#pragma unroll
    for (int n = 0; n < NG; ++n) {
#pragma unroll
        for (int t = 0; t < DEC_SUB; ++t)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[t][n][c] *= scale_log2;
        if (!inside) {
            const int kc = key0 + (lane >> 2);
#pragma unroll
            for (int t = 0; t < DEC_SUB; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int key = kc + 16 * t + ((c >> 1) << 3);
                    if (key < start || key >= key_end) s[t][n][c] = -INFINITY;
                }
        }
        float mx[2], less[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            mx[j] = fmaxf(s[0][n][j], s[0][n][j + 2]);
#pragma unroll
            for (int t = 1; t < DEC_SUB; ++t) mx[j] = fmaxf(mx[j], fmaxf(s[t][n][j], s[t][n][j + 2]));
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], o));
            part.m[n][j] = mx[j];
            // (no key in sight: every weight 2^(-inf - 0) = 0; a score that is no number makes its head none)
            less[j] = mx[j] == -INFINITY ? 0.f : mx[j];
            part.l[n][j] = 0.f;
        }
#pragma unroll
        for (int t = 0; t < DEC_SUB; ++t) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[t][n][c] = ex2(s[t][n][c] - less[c & 1]);
                part.l[n][c & 1] += s[t][n][c];
            }
            p[t][n][0] = transpose_8x8(pack_bf16(s[t][n][0], s[t][n][1]));
            p[t][n][1] = transpose_8x8(pack_bf16(s[t][n][2], s[t][n][3]));
        }
    }
    // O^T = V^T P^T
#pragma unroll
    for (int i = 0; i < D / 16; ++i)
#pragma unroll
        for (int n = 0; n < NG; ++n) part.o[i][n][0] = part.o[i][n][1] = part.o[i][n][2] = part.o[i][n][3] = 0.f;
#pragma unroll
    for (int t = 0; t < DEC_SUB; ++t) {
        if (t > 0 && !whole && t >= tiles) continue;
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            unsigned a[4];
            ldmatrix_x4_trans_at(a, smem + t * 2 * TILE + TILE + at.v_at(i));
#pragma unroll
            for (int n = 0; n < NG; ++n) mma_bf16(part.o[i][n], a, p[t][n][0], p[t][n][1]);
        }
        __syncwarp();
        done(t);
    }
}

// Where a request's keys lie in tiles and pieces.
struct DecRange {
    int kv_len, start, tile_first, tile_last, npieces;   // (tile_last: exclusive)
};
__device__ __forceinline__ DecRange dec_range(int position, int window, int piece_tiles, int max_pieces) {
    DecRange r;
    r.kv_len = position + 1;
    r.start = (window > 0 && r.kv_len > window) ? r.kv_len - window : 0;
    r.tile_first = r.start >> 4;
    r.tile_last = (r.kv_len + 15) >> 4;
    // (a caller whose max_pieces is too small for this request loses keys, but nothing is
    // read or written outside the scratch)
    r.npieces = min((r.tile_last - r.tile_first + piece_tiles - 1) / piece_tiles, max_pieces);
    return r;
}

// Writes channels 16 i0 .. 16 (i0 + NI) of a finished piece: the output if the request has one piece, else the
// unnormalised accumulator and (max, sum) to the scratch.
template <int D, int NG, int NI>
__device__ __forceinline__ void dec_write_piece(const float (&o)[NI][NG][4], const float (&m)[NG][2], float (&l)[NG][2], int i0,
                                                bool write_ml, int npieces, size_t head0, int max_pieces, int piece, int G,
                                                float* part_o, float* part_ml, bf16* out_row, int lane) {
#pragma unroll
    for (int n = 0; n < NG; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) l[n][j] += __shfl_xor_sync(0xffffffffu, l[n][j], x);
            const int g = 8 * n + ((lane & 3) << 1) + j;
            if (g >= G) continue;
            const int d = 16 * i0 + (lane >> 2);
            if (npieces == 1) {
                const float inv = 1.f / l[n][j];
                bf16* dst = out_row + (size_t)g * D + d;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    dst[16 * i] = __float2bfloat16_rn(o[i][n][j] * inv);
                    dst[16 * i + 8] = __float2bfloat16_rn(o[i][n][j + 2] * inv);
                }
            } else {
                const size_t p = (head0 + g) * max_pieces + piece;
                float* dst = part_o + p * D + d;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    dst[16 * i] = o[i][n][j];
                    dst[16 * i + 8] = o[i][n][j + 2];
                }
                if (write_ml && lane < 4) *reinterpret_cast<float2*>(part_ml + p * 2) = make_float2(m[n][j], l[n][j]);
            }
        }
}

// Which piece of which request and kv head block `number` takes: a head's pieces one after another, but where no request has more
// than two, the first ones, which are whole, before the second ones, which are not: the longest come first, and the last round of the
// SMs is short (64 requests of 300 keys, 16 and 32 query heads on 8: 20.2 and 22.2 -> 18.4 and 20.2 us).
__device__ __forceinline__ void dec_locate(int number, int Hk, int max_pieces, int& b, int& hk, int& piece) {
    if (max_pieces == 2) {
        const int half = (int)gridDim.x >> 1;
        piece = number >= half;
        number -= piece * half;
        b = number / Hk;
        hk = number % Hk;
    } else {
        const int per_request = Hk * max_pieces;
        b = number / per_request;
        hk = (number % per_request) / max_pieces;
        piece = number % max_pieces;
    }
}

// A warp (a block of its own) per piece, RING tiles of K and V in shared memory.
template <int D, int NG, int RING>
__global__ void __launch_bounds__(32)
paged_decode_attention_kernel(const bf16* __restrict__ q, int q_row_stride, const bf16* __restrict__ k_pool,
                              const bf16* __restrict__ v_pool, const int* __restrict__ block_table,
                              int max_blocks, const int* __restrict__ token_rows,
                              const int* __restrict__ seq_of_token, const int* __restrict__ positions,
                              float* __restrict__ part_o, float* __restrict__ part_ml, int max_pieces,
                              bf16* __restrict__ out, int out_row_stride, float scale_log2, int window,
                              int H, int Hk, int S, int piece_tiles, int early_ok) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int TILE_BYTES = 16 * D * 2;
    const int lane = threadIdx.x;
    int b, hk, piece;
    dec_locate((int)blockIdx.x, Hk, max_pieces, b, hk, piece);
    const int G = H / Hk;
    // The step's description was copied to the device before any kernel of the
    // step ran, so it may be read before the wait on earlier kernels.
    const int row_tok = token_rows ? token_rows[b] : b;
    const int seq = seq_of_token[row_tok];
    const DecRange range = dec_range(positions[row_tok], window, piece_tiles, max_pieces);
    const int kv_len = range.kv_len;
    if (piece >= range.npieces) return;
    const int tile_begin = range.tile_first + piece * piece_tiles;
    const int count = min(piece_tiles, range.tile_last - tile_begin);
    const int* bt = block_table + (size_t)seq * max_blocks;
    // lane j holds where the warp's j-th tile lies
    int my_rows = 0;
    if (lane < count) my_rows = dec_tile_rows(bt, tile_begin + lane, hk, Hk, S);
    const DecLane<D> at(lane);
    const bf16 *k_lane = k_pool + lane * 8, *v_lane = v_pool + lane * 8;
    const unsigned smem = (unsigned)__cvta_generic_to_shared(smem_raw);
    // The tiles asked for first hold keys and values of earlier steps, unless they reach the
    // request's newest position (which the kernel before this one has just written, or is
    // still writing): only then do they have to wait for that kernel.
    // (`early_ok` is 0 when a request brings several tokens in this step: then the kernel before this
    // one has written more than the newest position, and nothing is asked for before the wait)
    const bool early = early_ok && ((tile_begin + min(RING, count)) << 4) <= kv_len - 1;
    auto issue = [&](int j, unsigned slot) {
        const int rows = __shfl_sync(0xffffffffu, my_rows, j & 31);
        if (j < count) dec_ask_tile<D>(slot, k_lane, v_lane, rows, at);
        cp_async_commit();   // (one group a tile, empty past the last: the waits below count groups)
    };
    if (early)
        for (int j = 0; j < RING; ++j) issue(j, smem + j * 2 * TILE_BYTES);
    pdl_wait();
    pdl_trigger();
    if (!early)
        for (int j = 0; j < RING; ++j) issue(j, smem + j * 2 * TILE_BYTES);

    unsigned qf[D / 16][NG][2];
    dec_load_queries<D, NG>(qf, q + (size_t)row_tok * q_row_stride + (size_t)hk * G * D, G, lane);
    DecPart<D, NG> part, total;
    total.clear();
    unsigned next = smem;   // where the next sub-piece lies in the ring
    for (int i = 0; i < count; i += DEC_SUB) {
        cp_async_wait<RING - DEC_SUB>();
        __syncwarp();
        dec_sub_piece<D, NG>(part, qf, next, at, min(DEC_SUB, count - i), (tile_begin + i) << 4, range.start, kv_len, scale_log2, lane,
                             [&](int t) { issue(i + t + RING, next + t * 2 * TILE_BYTES); });
        next = next == smem + (RING - DEC_SUB) * 2 * TILE_BYTES ? smem : next + DEC_SUB * 2 * TILE_BYTES;
#pragma unroll
        for (int n = 0; n < NG; ++n)
#pragma unroll
            for (int j = 0; j < 2; ++j) {   // (onto nothing, m = -inf, the sub-piece comes out as it is)
                float fa, fb;
                fold_factors(total.m[n][j], part.m[n][j], fa, fb);
                total.l[n][j] = fold_add(total.l[n][j], fa, part.l[n][j], fb);
#pragma unroll
                for (int c = 0; c < D / 16; ++c) {
                    total.o[c][n][j] = fold_add(total.o[c][n][j], fa, part.o[c][n][j], fb);
                    total.o[c][n][j + 2] = fold_add(total.o[c][n][j + 2], fa, part.o[c][n][j + 2], fb);
                }
            }
    }
    cp_async_wait<0>();
    dec_write_piece<D, NG, D / 16>(total.o, total.m, total.l, 0, true, range.npieces, (size_t)b * H + hk * G, max_pieces, piece, G,
                                   part_o, part_ml, out + (size_t)row_tok * out_row_stride + (size_t)hk * G * D, lane);
}

// A block of eight warps per piece of 256 keys, each a sub-piece: when the step has so few pieces that every one finds an
// SM of its own, the time of a warp that walks a piece alone is what the step waits for.
#define DEC_SPLIT_WARPS 8
template <int D, int NG>
__global__ void __launch_bounds__(DEC_SPLIT_WARPS * 32)
paged_decode_split_kernel(const bf16* __restrict__ q, int q_row_stride, const bf16* __restrict__ k_pool,
                          const bf16* __restrict__ v_pool, const int* __restrict__ block_table,
                          int max_blocks, const int* __restrict__ token_rows,
                          const int* __restrict__ seq_of_token, const int* __restrict__ positions,
                          float* __restrict__ part_o, float* __restrict__ part_ml, int max_pieces,
                          bf16* __restrict__ out, int out_row_stride, float scale_log2, int window,
                          int H, int Hk, int S, int early_ok) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int TILE_BYTES = 16 * D * 2, PIECE_TILES = DEC_SPLIT_WARPS * DEC_SUB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int number = (int)blockIdx.x, per_request = Hk * max_pieces;
    const int b = number / per_request, hk = (number % per_request) / max_pieces, piece = number % max_pieces;
    const int G = H / Hk;
    const int row_tok = token_rows ? token_rows[b] : b;
    const int seq = seq_of_token[row_tok];
    const DecRange range = dec_range(positions[row_tok], window, PIECE_TILES, max_pieces);
    const int kv_len = range.kv_len;
    if (piece >= range.npieces) return;  // (the whole block)
    const int piece_begin = range.tile_first + piece * PIECE_TILES;
    const int piece_count = min(PIECE_TILES, range.tile_last - piece_begin);
    const int subs = (piece_count + DEC_SUB - 1) / DEC_SUB;
    const int tile_begin = piece_begin + warp * DEC_SUB;
    const int count = min(max(piece_count - warp * DEC_SUB, 0), DEC_SUB);
    int my_rows = 0;
    if (lane < count) my_rows = dec_tile_rows(block_table + (size_t)seq * max_blocks, tile_begin + lane, hk, Hk, S);
    const DecLane<D> at(lane);
    const unsigned smem = (unsigned)__cvta_generic_to_shared(smem_raw) + warp * DEC_SUB * 2 * TILE_BYTES;
    const bool early = early_ok && ((tile_begin + count) << 4) <= kv_len - 1;
    auto issue_all = [&]() {
#pragma unroll
        for (int j = 0; j < DEC_SUB; ++j) {
            const int rows = __shfl_sync(0xffffffffu, my_rows, j);
            if (j < count) dec_ask_tile<D>(smem + j * 2 * TILE_BYTES, k_pool + lane * 8, v_pool + lane * 8, rows, at);
        }
        cp_async_commit();
    };
    if (early) issue_all();
    pdl_wait();
    pdl_trigger();
    if (!early) issue_all();
    unsigned qf[D / 16][NG][2];
    dec_load_queries<D, NG>(qf, q + (size_t)row_tok * q_row_stride + (size_t)hk * G * D, G, lane);

    DecPart<D, NG> part;
    part.clear();
    cp_async_wait<0>();
    __syncwarp();
    if (count > 0)
        dec_sub_piece<D, NG>(part, qf, smem, at, count, tile_begin << 4, range.start, kv_len, scale_log2, lane, [](int) {});

    // fold the sub-pieces: every thread's registers through shared memory, every warp its share of the channels
    constexpr int REGS = D / 16 * NG * 4, NI = D / 16 > DEC_SPLIT_WARPS ? D / 16 / DEC_SPLIT_WARPS : 1;   // (NI: tiles of 16 channels a warp)
    float* ex = reinterpret_cast<float*>(smem_raw);      // [sub-piece][REGS + 4 NG][lane]
    __syncthreads();
    if (warp < subs) {
        float* mine = ex + (size_t)warp * (REGS + 4 * NG) * 32 + lane;
#pragma unroll
        for (int r = 0; r < REGS; ++r) mine[r * 32] = part.o[r / (4 * NG)][r / 4 % NG][r % 4];
#pragma unroll
        for (int r = 0; r < 2 * NG; ++r) {
            mine[(REGS + r) * 32] = part.m[r >> 1][r & 1];
            mine[(REGS + 2 * NG + r) * 32] = part.l[r >> 1][r & 1];
        }
    }
    __syncthreads();
    if (warp * NI >= D / 16) return;
    float o[NI][NG][4], m[NG][2], l[NG][2];
    const float* from = ex + lane;
#pragma unroll
    for (int r = 0; r < NI * NG * 4; ++r) o[r / (4 * NG)][r / 4 % NG][r % 4] = from[(warp * NI * NG * 4 + r) * 32];
#pragma unroll
    for (int r = 0; r < 2 * NG; ++r) {
        m[r >> 1][r & 1] = from[(REGS + r) * 32];
        l[r >> 1][r & 1] = from[(REGS + 2 * NG + r) * 32];
    }
    for (int s = 1; s < subs; ++s) {
        from += (REGS + 4 * NG) * 32;
#pragma unroll
        for (int r = 0; r < 2 * NG; ++r) {
            const int n = r >> 1, j = r & 1;
            float fa, fb;
            fold_factors(m[n][j], from[(REGS + r) * 32], fa, fb);
            l[n][j] = fold_add(l[n][j], fa, from[(REGS + 2 * NG + r) * 32], fb);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const float* p = from + ((warp * NI + i) * NG + n) * 4 * 32;
                o[i][n][j] = fold_add(o[i][n][j], fa, p[j * 32], fb);
                o[i][n][j + 2] = fold_add(o[i][n][j + 2], fa, p[(j + 2) * 32], fb);
            }
        }
    }
    dec_write_piece<D, NG, NI>(o, m, l, warp * NI, warp == 0, range.npieces, (size_t)b * H + hk * G, max_pieces, piece, G, part_o,
                               part_ml, out + (size_t)row_tok * out_row_stride + (size_t)hk * G * D, lane);
}

// Joins the pieces of requests that have several: one block per (request, head).  Each of its four warps adds every
// fourth piece, in piece order, and the warps' sums are added in warp order: the order depends on the number of pieces
// alone.  (Joining in the kernel above, by whichever block of a request finishes last, took as long or longer: its fence
// and counter come one after another with the join, while this kernel's launch overlaps.)
#define JOIN_MAX_PIECES 1024
#define JOIN_AHEAD 8   // pieces whose values a thread asks for at a time, the first ones before it knows their weights
template <int D>
__global__ void __launch_bounds__(128)
paged_decode_join_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                         int max_pieces, const int* __restrict__ token_rows,
                         const int* __restrict__ positions, bf16* __restrict__ out,
                         int out_row_stride, int window, int H, int piece_tiles) {
    constexpr int E = D / 32;   // channels a lane
    __shared__ float2 wl[JOIN_MAX_PIECES];
    __shared__ float top[4];
    __shared__ float sums[4][D + 1];
    const int b = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_tok = token_rows ? token_rows[b] : b;
    const int npieces = dec_range(positions[row_tok], window, piece_tiles, max_pieces).npieces;
    pdl_wait();  // on every path: a grid that ends without waiting would let its successor run ahead of its predecessor
    pdl_trigger();
    if (npieces <= 1) return;  // written by the first pass
    const size_t p0 = ((size_t)b * H + h) * max_pieces;
    const float* po = part_o + p0 * D + lane * E;
    float v[JOIN_AHEAD][E];
    auto ask = [&](int s0) {
#pragma unroll
        for (int u = 0; u < JOIN_AHEAD; ++u) {
            const int s = s0 + 4 * u;
            if (s >= npieces) continue;
#pragma unroll
            for (int e = 0; e < E; e += 2) {   // (the scratch need only be aligned to 8 bytes)
                const float2 x = *reinterpret_cast<const float2*>(po + (size_t)s * D + e);
                v[u][e] = x.x;
                v[u][e + 1] = x.y;
            }
        }
    };
    ask(warp);
    // weights of the pieces, w_s = 2^(m_s - M)
    float M = -INFINITY;
    for (int s = threadIdx.x; s < npieces; s += 128) {
        wl[s] = *reinterpret_cast<const float2*>(part_ml + (p0 + s) * 2);
        M = fmaxf(M, wl[s].x);
    }
    M = warp_max(M);
    if (lane == 0) top[warp] = M;
    __syncthreads();
    M = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
    for (int s = threadIdx.x; s < npieces; s += 128) wl[s].x = wl[s].x == -INFINITY ? 0.f : exp2f(wl[s].x - M);
    __syncthreads();
    float O[E], L = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) O[e] = 0.f;
    for (int s0 = warp; s0 < npieces; s0 += 4 * JOIN_AHEAD) {
        if (s0 != warp) ask(s0);
#pragma unroll
        for (int u = 0; u < JOIN_AHEAD; ++u) {
            const int s = s0 + 4 * u;
            if (s >= npieces) continue;
            const float2 w = wl[s];
            L += w.x * w.y;
#pragma unroll
            for (int e = 0; e < E; ++e) O[e] += w.x * v[u][e];
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) sums[warp][lane * E + e] = O[e];
    if (lane == 0) sums[warp][D] = L;
    __syncthreads();
    const int d = threadIdx.x;
    if (d >= D) return;
    const float l = sums[0][D] + sums[1][D] + sums[2][D] + sums[3][D];
    const float o = sums[0][d] + sums[1][d] + sums[2][d] + sums[3][d];
    out[(size_t)row_tok * out_row_stride + (size_t)h * D + d] = __float2bfloat16_rn(o * (1.f / l));
}

// Scratch a launch needs, in floats: accumulators [requests, H, max_pieces, D] then
// (max, sum) [requests, H, max_pieces, 2].  Every element is written before it is
// read; nothing needs clearing.
extern "C" long long vx_paged_decode_scratch_floats(int requests, int H, int D, int max_pieces) {
    return (long long)requests * H * max_pieces * (D + 2);
}

static int dec_sm_count() {
    static int sms[VX_MAX_DEVICES];
    return vx_sm_count(sms);
}

// shared memory of `tiles` tiles of K and V
template <int D>
static size_t dec_smem(int tiles) { return (size_t)tiles * 2 * 16 * D * 2; }

// Both kernels of a head size at its first call on a device (the attributes belong
// to a device's copy of the function), whichever that call needs: a later call
// may come from inside a stream capture with a step of another size.  First calls are
// not made from several host threads at once.
template <int D, int NG>
static int configure_decode() {
    static bool configured[VX_MAX_DEVICES];
    const int dev = vx_current_device();
    if (dev < 0) return VX_ERR_LIMIT;
    if (configured[dev]) return VX_OK;
    const cudaFuncAttribute most = cudaFuncAttributeMaxDynamicSharedMemorySize, carveout = cudaFuncAttributePreferredSharedMemoryCarveout;
    cudaError_t e = cudaFuncSetAttribute(paged_decode_split_kernel<D, NG>, most, (int)dec_smem<D>(DEC_SPLIT_WARPS * DEC_SUB));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(paged_decode_attention_kernel<D, NG, 2 * DEC_SUB>, most, (int)dec_smem<D>(2 * DEC_SUB));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(paged_decode_attention_kernel<D, NG, 2 * DEC_SUB>, carveout, DEC_CARVEOUT);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(paged_decode_split_kernel<D, NG>, carveout, DEC_CARVEOUT);
    if (e != cudaSuccess) return (int)e;
    configured[dev] = true;
    return VX_OK;
}

template <int D, int NG>
static int launch_decode(const bf16* q, int q_row_stride, const bf16* k_pool, const bf16* v_pool,
                         const int* block_table, int max_blocks, const int* token_rows,
                         const int* seq_of_token, const int* positions, float* scratch, int max_pieces,
                         bf16* out, int out_row_stride, float scale, int window, int requests, int H, int Hk,
                         int S, int piece_tiles, int early_ok, int shape, cudaStream_t stream) {
    const int ready = configure_decode<D, NG>();
    if (ready != VX_OK) return ready;
    float* part_o = scratch;
    float* part_ml = scratch ? scratch + (size_t)requests * H * max_pieces * D : nullptr;
    const int pieces = requests * Hk * max_pieces;
    const bool splits = piece_tiles == DEC_SPLIT_WARPS * DEC_SUB;
    if (shape == 0) shape = splits && pieces <= dec_sm_count() ? 8 : 1;
    if (shape == 8 && splits)
        VX_LAUNCH_K(VX_K_ATTENTION, (paged_decode_split_kernel<D, NG>), pieces, DEC_SPLIT_WARPS * 32,
                    dec_smem<D>(DEC_SPLIT_WARPS * DEC_SUB), stream, q, q_row_stride, k_pool, v_pool, block_table, max_blocks,
                    token_rows, seq_of_token, positions, part_o, part_ml, max_pieces, out, out_row_stride, scale * LOG2E, window,
                    H, Hk, S, early_ok);
    else if (shape == 1)
        VX_LAUNCH_K(VX_K_ATTENTION, (paged_decode_attention_kernel<D, NG, 2 * DEC_SUB>), pieces, 32, dec_smem<D>(2 * DEC_SUB), stream, q,
                    q_row_stride, k_pool, v_pool, block_table, max_blocks, token_rows, seq_of_token, positions, part_o, part_ml,
                    max_pieces, out, out_row_stride, scale * LOG2E, window, H, Hk, S, piece_tiles, early_ok);
    else
        return VX_ERR_SHAPE;
    VX_LAUNCH_CHECK();
    if (max_pieces > 1) {
        dim3 jgrid(requests, H);
        VX_LAUNCH_K(VX_K_JOIN, (paged_decode_join_kernel<D>), jgrid, 128, 0, stream, part_o, part_ml, max_pieces,
                  token_rows, positions, out, out_row_stride, window, H, piece_tiles);
        VX_LAUNCH_CHECK();
    }
    return VX_OK;
}

// One query token per entry.  `token_rows[i]` is the token row (in q, out,
// seq_of_token, positions) of entry i, or null when entry i is row i; several
// entries may be tokens of one request (a short prompt portion, token by token).
// `early_ok`: every entry is its request's only new token of this step (then a warp
// may ask for keys and values of earlier positions before the kernel before it ends).
// `max_pieces` bounds the pieces of any request: ceil(ceil(max keys / 16) / piece_tiles)
// (one more with a window that does not start on a tile's edge); `scratch` holds
// vx_paged_decode_scratch_floats(...) floats (may be null when max_pieces is 1).
// `shape`: 0 lets the sizes choose; 8: a block of eight warps a piece (pieces of 16 tiles); 1: a warp a piece.
extern "C" int vx_paged_decode_attention_shape(const void* q, int q_row_stride, const void* k_pool,
                                               const void* v_pool, const int* block_table, int max_blocks,
                                               const int* token_rows, const int* seq_of_token,
                                               const int* positions, float* scratch, int max_pieces, void* out,
                                               int out_row_stride, float scale, int window, int requests, int H,
                                               int Hk, int D, int S, int piece_tiles, int early_ok, int shape, cudaStream_t stream) {
    if (requests <= 0) return VX_OK;
    if (H <= 0 || Hk <= 0 || H % Hk || H / Hk > 16 || S <= 0 || S % 16 || window < 0) return VX_ERR_SHAPE;
    if (piece_tiles <= 0 || piece_tiles > 32 || max_pieces <= 0 || (max_pieces > 1 && !scratch)) return VX_ERR_SHAPE;
    if (Hk > 65535 || requests > 65535 || max_pieces > JOIN_MAX_PIECES) return VX_ERR_LIMIT;
    if ((long long)requests * Hk * max_pieces > (1ll << 30)) return VX_ERR_LIMIT;   // pieces are numbered in an int
    if ((q_row_stride & 1) || (((uintptr_t)q) & 3) || (out_row_stride & 1) || (((uintptr_t)out) & 3)) return VX_ERR_ALIGN;
#define DEC_GO(DIM, NG)                                                                                                \
    launch_decode<DIM, NG>((const bf16*)q, q_row_stride, (const bf16*)k_pool, (const bf16*)v_pool, block_table, max_blocks, \
                           token_rows, seq_of_token, positions, scratch, max_pieces, (bf16*)out, out_row_stride, scale, \
                           window, requests, H, Hk, S, piece_tiles, early_ok, shape, stream)
    if (D == 128) return H / Hk <= 8 ? DEC_GO(128, 1) : DEC_GO(128, 2);
    if (D == 64) return H / Hk <= 8 ? DEC_GO(64, 1) : DEC_GO(64, 2);
#undef DEC_GO
    return VX_ERR_SHAPE;
}

extern "C" int vx_paged_decode_attention(const void* q, int q_row_stride, const void* k_pool,
                                         const void* v_pool, const int* block_table, int max_blocks,
                                         const int* token_rows, const int* seq_of_token,
                                         const int* positions, float* scratch, int max_pieces, void* out,
                                         int out_row_stride, float scale, int window, int requests, int H,
                                         int Hk, int D, int S, int piece_tiles, int early_ok, cudaStream_t stream) {
    return vx_paged_decode_attention_shape(q, q_row_stride, k_pool, v_pool, block_table, max_blocks, token_rows, seq_of_token,
                                           positions, scratch, max_pieces, out, out_row_stride, scale, window, requests, H, Hk,
                                           D, S, piece_tiles, early_ok, 0, stream);
}

// ----------------------------------------------------------------------------
// The variant that allocates nothing (declared and described in no_alloc.h).
#include "no_alloc.h"

// The scratch itself.  In host code this name is only a handle for the runtime's
// symbol lookup, never a device address: the address comes from
// cudaGetSymbolAddress below.
static __device__ __align__(256) float g_decode_static_scratch[VX_DECODE_STATIC_SCRATCH_FLOATS];

static float* g_decode_static_ptr[VX_MAX_DEVICES];  // device address of the array, per device

extern "C" long long vx_paged_decode_static_max_floats(void) { return VX_DECODE_STATIC_SCRATCH_FLOATS; }

extern "C" int vx_paged_decode_attention_static(const void* q, int q_row_stride, const void* k_pool,
                                                const void* v_pool, const int* block_table, int max_blocks,
                                                const int* token_rows, const int* seq_of_token,
                                                const int* positions, int max_splits, void* out,
                                                int out_row_stride, float scale, int window, int requests,
                                                int H, int Hk, int D, int S, int chunk_tiles,
                                                cudaStream_t stream) {
    if (requests <= 0) return VX_OK;
    if (H <= 0 || D <= 0 || max_splits <= 0) return VX_ERR_SHAPE;
    if (vx_paged_decode_scratch_floats(requests, H, D, max_splits) > (long long)VX_DECODE_STATIC_SCRATCH_FLOATS)
        return VX_ERR_LIMIT;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= VX_MAX_DEVICES) return VX_ERR_LIMIT;
    if (!g_decode_static_ptr[dev]) {
        // set-up, once per device, with that device current
        float* p = nullptr;
        e = cudaGetSymbolAddress((void**)&p, g_decode_static_scratch);
        if (e != cudaSuccess) return (int)e;
        if (!p) return VX_ERR_ALIGN;
        g_decode_static_ptr[dev] = p;
    }
    // The kernel before this one in the stream is the caller's, not this library's: it may
    // write what these kernels read ahead of their wait on it when launched programmatically
    // (the step's description, keys and values of earlier positions).  So: plain stream order.
    vx_pdl_suppress(1);
    const int rc = vx_paged_decode_attention(q, q_row_stride, k_pool, v_pool, block_table, max_blocks, token_rows,
                                             seq_of_token, positions, g_decode_static_ptr[dev], max_splits, out,
                                             out_row_stride, scale, window, requests, H, Hk, D, S, chunk_tiles, 1, stream);
    vx_pdl_suppress(0);
    return rc;
}
