// Shared helpers: bf16 conversion with the reference's rounding
// (src/cuda/cuda_internal.h:21-40 in o1.c: RNE by integer add, no NaN
// special case), 128-bit vector types, error slot, stream handling.
// On the device the rounding is the hardware conversion (cvt.rn.bf16.f32 /
// cvt.rn.bf16x2.f32: one instruction instead of five per value; the epilogues
// and elementwise kernels round several times per element).  It gives the
// same result as the integer form for every finite input and infinity; only
// NaN payloads differ (canonical NaN instead of a shifted payload).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

namespace o1 {

__host__ __device__ __forceinline__ float bf16_to_f32(uint16_t b) {
    uint32_t u = ((uint32_t)b) << 16;
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    __builtin_memcpy(&f, &u, 4);
    return f;
#endif
}
__host__ __device__ __forceinline__ uint16_t f32_to_bf16(float f) {
#ifdef __CUDA_ARCH__
    uint16_t r;
    asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(r) : "f"(f));
    return r;
#else
    uint32_t u;
    __builtin_memcpy(&u, &f, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
#endif
}
__host__ __device__ __forceinline__ float bf16_round(float f) {
    return bf16_to_f32(f32_to_bf16(f));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float bf16lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

// Both values rounded to bf16 (one conversion instead of two).
__device__ __forceinline__ void bf16_round2(float& a, float& b) {
    const uint32_t p = pack_bf16x2(a, b);
    a = bf16lo(p);
    b = bf16hi(p);
}

// GELU, tanh form: 0.5 v (1 + tanh u) with u = sqrt(2/pi) (v + 0.044715 v^3).  (1 + tanh u) / 2 = 1 / (1 + e^-2u), so
// one exponential and one reciprocal do, without tanhf's branches and without the cancellation of 1 + tanh u for u < 0.  e^-2u is
// taken as 2^t, t = -2 log2(e) u: instructions count, an epilogue of
// 128 x 128 values issued some 45 for each with expf and a division (the tower at 520 patches 2054 -> 2002 us).
__device__ __forceinline__ float gelu_tanh(float v) {
    const float t = v * __fmaf_rn(-0.102943240f, v * v, -2.302208198f);
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return v * r;
}

// One component of the vision tower's fp32 rotary, x cos + partner sin (the partner negated in the first half of a head),
// with its roundings written out: the stand-alone pass and the projection's epilogue give the same bits.
__device__ __forceinline__ float rope_f32(float x, float c, float partner, float s) {
    return __fmaf_rn(x, c, __fmul_rn(partner, s));
}

// ---- launches that overlap their start with the end of the kernel before them
// A forward is a chain of some ten launches per block, and at small sizes the time between two of them (the drain of
// one grid, the launch of the next, its barrier set-up) is a sizeable part of both.  launch_chained() lets the next
// grid be placed as soon as every block of this one has called grid_dep_launch(); its blocks set themselves up and stop
// in grid_dep_wait() until this grid has ended and its writes are visible.  Every kernel launched this way calls
// grid_dep_wait() in all its threads before it touches memory that another kernel writes or reads.
// Only up to OVERLAP_ROWS rows: with long kernels the early blocks cost more than they save.  With against without: a
// guided step of 296-row branches 10.95 / 11.38 ms, the tower at 520 rows 2.51 / 2.72 ms and at 4096 rows 9.14 / 9.28 ms, a
// block of 1280 rows 521 / 540 us; but a block of 4352 rows 1738 / 1712 us and of 16640 rows 9.52 / 9.25 ms.
static constexpr long OVERLAP_ROWS = 4096;
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A kernel that has failed (a wait ran out) leaves its code in the device's error word, and those after it store nothing.
// A chained kernel reads the word twice: early, beside its set-up, to do nothing at all after a failure that lies behind; and,
// since the kernels before it may still be running then, once more after grid_dep_wait(), in the threads that store, where
// the wait for the first result hides the read.
__device__ __forceinline__ int error_word(const int* err) { return *reinterpret_cast<const volatile int*>(err); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
[[nodiscard]] inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster,
                                  long rows, const A&... args) {
    cudaLaunchAttribute at[2];
    int n = 0;
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
        ++n;
    }
    if (rows <= OVERLAP_ROWS) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = at; cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    if (e != cudaSuccess) cudaGetLastError();     // the caller reports it: the next call's check must not find it again
    return e;
}

bool launch_ok(cudaError_t e, const char* what);     // sets the error text "<what>: ..." when e is one

// ---- process-wide state (one stream, one error buffer: the reference's
// primitive ABI has no stream argument and reports through a message buffer)
cudaStream_t current_stream();
char* errbuf();             // 512 bytes
void set_error(const char* fmt, ...);
int* device_failed_word();  // one int of mapped host memory per device, beside the error word (see lora.cu), or NULL
int* device_error_word();   // per-device int set by kernels whose bounded waits ran out
int sm_count();

#define O1_CUDA_OK(call, what)                                                     \
    do {                                                                           \
        cudaError_t e__ = (call);                                                  \
        if (e__ != cudaSuccess) o1::set_error("%s: %s", what, cudaGetErrorString(e__)); \
    } while (0)

}  // namespace o1
