// Shared helpers for the cinnamon_b200 CUDA library (sm_100a only).
#pragma once
#include <atomic>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>
#include <cstdio>
#include <cstdarg>

// ---- status codes returned by every extern "C" entry point -----------------
#define CINN_OK 0
#define CINN_ERR_INVALID 1      // bad argument (null pointer, shape, alignment, dtype)
#define CINN_ERR_CUDA 2         // a CUDA runtime/driver call failed
#define CINN_ERR_UNSUPPORTED 3  // valid request that this build cannot serve
#define CINN_ERR_DEVICE 4       // a kernel reported a device-side problem (bounded wait ran out)

// dtype tags of the C-ABI
#define CINN_BF16 0
#define CINN_F32 1
#define CINN_F16 2
#define CINN_F32_BF16 3   // GEMM output only: fp32 storage of the value rounded to bf16

// division flavour of the quantisers
#define CINN_DIV_FULL 0   // PTX div.full.f32: what Triton emits for the reference kernels on a GPU
#define CINN_DIV_RN 1     // IEEE round-to-nearest: what a CPU restatement computes

namespace cinn {

void set_error(const char* fmt, ...);

#define CINN_CHECK_ARG(cond, ...)                      \
    do {                                               \
        if (!(cond)) {                                 \
            cinn::set_error(__VA_ARGS__);              \
            return CINN_ERR_INVALID;                   \
        }                                              \
    } while (0)

#define CINN_CHECK_CUDA(expr)                                                          \
    do {                                                                               \
        cudaError_t _e = (expr);                                                       \
        if (_e != cudaSuccess) {                                                       \
            cinn::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),    \
                            __FILE__, __LINE__);                                       \
            return CINN_ERR_CUDA;                                                      \
        }                                                                              \
    } while (0)

// after every launch, and after nothing else: it also counts it (cinn_launch_count)
extern std::atomic<int64_t> g_launches;
#define CINN_CHECK_LAUNCH()                                          \
    do {                                                             \
        CINN_CHECK_CUDA(cudaGetLastError());                         \
        cinn::g_launches.fetch_add(1, std::memory_order_relaxed);    \
    } while (0)

// Programmatic dependent launch.  A kernel launched by launch_dependent may start while the one before it on the stream is
// still running, as soon as every block of that one has called pdl_trigger (or has ended); nothing it reads or writes in
// global memory may come before its pdl_wait, which returns when the kernel before has finished and its writes are visible.
// What is won is the launch latency and the prologue, which between kernels of 3 - 10 us are a quarter of the time.
// Two conditions on every kernel that triggers:
//   - It triggers after its own pdl_wait.  Whatever starts behind it then finds all that came before it done, which the quantisers that
//     work beside the kernel ahead of them build on: they read and write before they wait, and wait before they end.
//   - With tensor memory it triggers from the warp that allocates, after the allocation.  The kernels behind allocate before they wait: a block
//     that triggered first could find its columns taken by one that waits for its end, and neither would get on.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// Lets a kernel use up to `bytes` of dynamic shared memory, once per device.  The limit belongs to the function, not to a
// launch or a thread: it is set to the most any launch can ask for, so that no thread lowers it under another one.
template <auto KERN>
inline int allow_smem_once(size_t bytes) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    CINN_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && (done.load(std::memory_order_acquire) >> dev & 1)) return CINN_OK;
    CINN_CHECK_CUDA(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (dev >= 0 && dev < 64) done.fetch_or(1ULL << dev, std::memory_order_release);
    return CINN_OK;
}

int sm_count();   // SMs of the current device (cached per device)

// The tiles of the experts' row ranges, on the device: first row and rows of each, how many there are; at most `max`
struct SegmentTiles { const int *src, *cnt, *n; int max; };

// launch_dependent if `early`, else a plain launch: the kernel starts when the one before it has ended.  Both leave an error
// where CINN_CHECK_LAUNCH finds it.
template <typename... P, typename... A>
inline cudaError_t launch_early_if(bool early, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    if (early) return launch_dependent(kern, grid, block, smem, st, static_cast<A&&>(args)...);
    kern<<<grid, block, smem, st>>>(static_cast<P>(args)...);
    return cudaPeekAtLastError();
}
// Whether a launch on this stream becomes a node of a graph (never on the null stream).  What an early start wins is the gap between two launches, and between a
// graph's nodes there is little of one.  us a replayed pass, quantisers, combine and row spread early and plain: linear forward and backward
// 4096 x 512 -> 2048 55.6 and 53.9, 512 x 512 -> 2048 23.8 and 22.9, 2048 x 2048 -> 8192 158.1 and 156.1, forward 100 x 768 -> 2688 8.0 and 7.5,
// serving layer of 64 tokens 79.5 and 77.1; the other way 300 x 512 -> 512 17.6 and 18.0, forward 4096 x 512 -> 2048 13.7 and 14.1, serving one
// token 46.3 and 47.1.
inline bool captured(cudaStream_t st) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    return st != nullptr && cudaStreamIsCapturing(st, &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
}
// Whether a quantiser of so many rows starts early.  Short ones gain the launch.  In front of a GEMM of long tiles an early start costs more than it
// wins, up to a tile's time: 403 x 4032 -> 12928 80 -> 96 us, 1824 x 6976 -> 8832 forward and backward 458 -> 470, 16384 x 7168 -> 18432 7020 ->
// 7130; in front of short ones it wins: 4096 x 512 -> 2048 16.4 -> 14.5, 32768 x 512 -> 1024 forward and backward 132 -> 129.
inline bool quantise_early(int64_t rows, int64_t length, cudaStream_t st) {
    return length <= 2048 && rows * length <= (int64_t)1 << 26 && !captured(st);
}

// ---- arithmetic shared by every quantiser ---------------------------------
constexpr float kFp8Max = 448.0f;
constexpr float kAmaxFloor = 1e-4f;   // 0x38D1B717

template <int DIV>
__device__ __forceinline__ float div_f32(float a, float b) {
    if constexpr (DIV == CINN_DIV_FULL) {
        float r;
        asm("div.full.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
        return r;
    } else {
        return __fdiv_rn(a, b);
    }
}

// amax (>= 0, NaN already dropped) -> scale.
// round_scale: 2^ceil(log2(amax/448)) with log2 evaluated by CUDA's fp32 log2f,
// rounded up by cvt.rpi and exponentiated by ex2.approx (exact for integers).
template <int DIV, bool ROUND>
__device__ __forceinline__ float scale_from_amax(float amax) {
    amax = fmaxf(amax, kAmaxFloor);
    float s = div_f32<DIV>(amax, kFp8Max);
    if constexpr (ROUND) {
        float lg = log2f(s);
        float e, r;
        asm("cvt.rpi.ftz.f32.f32 %0, %1;" : "=f"(e) : "f"(lg));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(e));
        s = r;
    }
    return s;
}

// Many elements are divided by one scale.  In the div.full.f32 flavour the quotient x / s is formed as
// x * rcp.approx(s) with the reciprocal taken once per scale: for every divisor in [2^-126, 2^126] (all scales these
// kernels produce: the amax has a floor of 1e-4 and is finite) that product has the very bits of
// div.full.f32(x, s), which cinn_selfcheck_division confirms on the GPU at hand for every 16-bit x and every
// scale a 16-bit amax can give.  The IEEE flavour divides element by element.
template <int DIV>
__device__ __forceinline__ float divisor_of(float s) {
    if constexpr (DIV == CINN_DIV_FULL) {
        float r;
        asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(s));
        return r;
    } else {
        return s;
    }
}

// x / s (d = divisor_of(s)), clamped from below.
template <int DIV>
__device__ __forceinline__ float scaled_clamped(float x, float d) {
    float y;
    if constexpr (DIV == CINN_DIV_FULL) y = __fmul_rn(x, d);
    else y = __fdiv_rn(x, d);
    // The reference clamps with max(y, -448) then min(., 448), both dropping a NaN operand.
    // Only the max is kept: it turns NaN into -448 as the reference does; the upper (and lower)
    // clamp is what the saturating e4m3 conversion that always follows does anyway.
    return fmaxf(y, -kFp8Max);
}

// two fp32 -> two e4m3 bytes (lo in bits 0-7, hi in bits 8-15), RNE, finite saturation
__device__ __forceinline__ uint16_t cvt_e4m3x2(float lo, float hi) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t cvt_e4m3x4(float a, float b, float c, float d) {
    return (uint32_t)cvt_e4m3x2(a, b) | ((uint32_t)cvt_e4m3x2(c, d) << 16);
}

// e4m3 byte -> fp32 (exact): via the hardware e4m3x2 -> f16x2 conversion
__device__ __forceinline__ float2 e4m3x2_to_float2(uint16_t v) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(v));
    __half2 h = *reinterpret_cast<__half2*>(&h2);
    return __half22float2(h);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float bf16_bits_to_float(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }

}  // namespace cinn
