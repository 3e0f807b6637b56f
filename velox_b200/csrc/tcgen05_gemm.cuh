// What the tcgen05 matrix-product kernels share: mbarrier and TMA wrappers, the
// shared-memory descriptor of a swizzled K-major tile, tcgen05.ld, and the host's
// tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"

#define TC_BM 128
#define TC_BK 64
#define TC_THREADS 192
#define TC_SPIN_LIMIT (1 << 24)
#define TC_ERR_PRODUCER 1
#define TC_ERR_MMA 2
#define TC_ERR_EPILOGUE 3

__device__ __forceinline__ unsigned tc_smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void tc_mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tc_mbar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// A bounded wait of one thread.
__device__ __forceinline__ bool tc_mbar_wait(unsigned bar, unsigned parity) {
    for (int i = 0; i < TC_SPIN_LIMIT; ++i)
        if (tc_mbar_try(bar, parity)) return true;
    return false;
}
// A bounded wait of a whole warp, with one answer for all its lanes.  A role that goes on as a warp (tc_elect, tcgen05.ld) waits this
// way: if lanes counted by themselves, a phase that ends as the limit does could let some of them through and send others away, and an
// elect.sync that names lanes which have left is undefined.
__device__ __forceinline__ bool tc_warp_wait(unsigned bar, unsigned parity) {
    for (int i = 0; i < TC_SPIN_LIMIT; ++i)
        if (__all_sync(0xffffffffu, tc_mbar_try(bar, parity))) return true;
    return false;
}
__device__ __forceinline__ void tc_tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// Shared-memory descriptor of a K-major tile with 128-byte swizzle: rows 128 bytes
// apart, groups of 8 rows 1024 bytes apart (the tile is exactly one swizzle atom
// wide), version 1, layout type 2 (128-byte swizzle).
// In two words: the upper one is the same for every tile.
#define TC_DESC_HI 0x40004040u
__device__ __forceinline__ unsigned tc_desc_lo(unsigned addr) { return ((addr >> 4) & 0x3FFF) | (1u << 16); }
// One lane of the warp, the same every time.  A role that one thread has (loads, products) is run by its whole warp, and the
// elected lane issues: its operands then stay in the warp's uniform registers.  Under `if (lane == 0)` every operand of every
// instruction is moved there first: gated products with short tiles took up to 1.3 times as long (777 x 6144 x 1024 on tiles of 160
// columns 21.1 us, 19.3 so; 2048 x 19456 x 2560 by pairs 155, 146; 2048 x 24576 x 4096 by pairs 294, 277; the votes of tc_warp_wait among that,
// 1 to 3 %).
__device__ __forceinline__ bool tc_elect() {
    unsigned p;
    asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
    return p != 0;
}
// STEPS products of 16 k each (32 bytes further along K inside the swizzle atom) from descriptors given by their lower words;
// the first adds to the accumulator if `add` is not 0, the others always.
template <int CG, int STEPS>
__device__ __forceinline__ void tc_mma_run(unsigned tmem_d, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned add) {
#pragma unroll
    for (int k = 0; k < STEPS; ++k) {
        if (CG == 2)
            asm volatile("{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
                         " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n}\n"
                         ::"r"(tmem_d), "r"(a_lo + 2 * k), "r"(b_lo + 2 * k), "r"(idesc), "r"(k ? 1u : add), "r"(TC_DESC_HI) : "memory");
        else
            asm volatile("{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %4, 0;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
                         " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n"
                         ::"r"(tmem_d), "r"(a_lo + 2 * k), "r"(b_lo + 2 * k), "r"(idesc), "r"(k ? 1u : add), "r"(TC_DESC_HI) : "memory");
    }
}
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_ld32(unsigned taddr, unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

typedef CUresult (*tc_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static tc_encode_fn tc_encoder() {
    static tc_encode_fn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (tc_encode_fn)p;
    }
    return fn;
}

// A [rows, K] bfloat16 matrix with row stride ld, read in boxes of box_rows x 64.
static bool tc_make_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows) {
    tc_encode_fn enc = tc_encoder();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {TC_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

