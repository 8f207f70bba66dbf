// Shared host/device helpers of librq_b200: status handling, dtype loads,
// small PTX wrappers.  sm_100a only.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/rq_b200.h"

namespace rq {

constexpr int kHeadDim = 128;       // the only head size the kernels are built for
constexpr int kHalfDim = 64;        // packed index bytes per (token, head)
constexpr int kSlotPerHead = 256;   // next_pow2(2 * (64 + 4)) bytes per head in a slot

// Thread-local message buffer behind rq_last_error().
char* error_buffer();
constexpr size_t kErrorBufferBytes = 512;

template <typename... Args>
inline int fail(int code, const char* fmt, Args... args) {
    snprintf(error_buffer(), kErrorBufferBytes, fmt, args...);
    return code;
}
inline int fail(int code, const char* msg) {
    snprintf(error_buffer(), kErrorBufferBytes, "%s", msg);
    return code;
}

inline int check_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return RQ_OK;
    return fail(RQ_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Raise a kernel's dynamic shared-memory limit; remembered per (kernel, device) so that later
// launches skip the driver call.  Safe to call before every launch and from several threads.
int ensure_smem_impl(const void* kernel, size_t bytes);
template <typename Kernel>
inline int ensure_smem(Kernel k, size_t bytes) {
    return ensure_smem_impl(reinterpret_cast<const void*>(k), bytes);
}

// SM count of the current device (148 on a B200), looked up once per device.
int sm_count();

// Launch with programmatic stream serialization: the kernel may be scheduled while the one before it on the stream
// drains, as soon as all of that kernel's CTAs have ended or called grid_launch_dependents().  It must not touch
// memory that earlier kernels write (or read, if it writes it) before grid_dependency_wait() returns.
template <typename... KArgs, typename... Args>
inline int launch_dependent(const char* what, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                            Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<Args&&>(args)...), what);
}

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

inline int dtype_bytes(int dt) { return dt == RQ_DTYPE_F32 ? 4 : 2; }

// Region offsets of one cache slot for H heads on this GPU.
struct SlotLayout {
    int k_idx, k_norm, v_idx, v_norm, payload_end, total;
};
__host__ __device__ inline SlotLayout slot_layout(int H) {
    SlotLayout l;
    l.k_idx = 0;
    l.k_norm = H * kHalfDim;
    l.v_idx = l.k_norm + H * 4;
    l.v_norm = l.v_idx + H * kHalfDim;
    l.payload_end = l.v_norm + H * 4;
    l.total = H * kSlotPerHead;
    return l;
}

// Programmatic dependent launch.  wait: every kernel before this one on the stream has completed (returns at once in
// a kernel launched without the attribute).  launch_dependents: the next kernel may be scheduled.  A kernel that
// waits before it lets the next one start makes everything older visible to the next one from its start.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- device helpers --------------------------------------------------------

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Pairs of fp32 values in one 64-bit register.  A packed operation takes the pipe as long as two scalar ones but
// one issue slot instead of two.  The assembler may contract a packed product and a packed sum into one operation.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void upk(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// ---- mbarrier (shared-memory barrier objects) -----------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// Wait until the phase with the given parity has completed.  Every wait in this library is
// bounded (about one second of SM clocks); false means the bound expired.
constexpr long long kWaitCycles = 2000000000LL;
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, long long limit_cycles) {
    const uint32_t addr = smem_u32(bar);
    long long start = 0;
    for (int spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
        if (spin == 0) start = clock64();
        else if (clock64() - start > limit_cycles) return false;
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    return mbar_wait_for(bar, parity, kWaitCycles);
}

}  // namespace rq
