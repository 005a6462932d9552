// Host-side plumbing shared by the .cu files: status codes, the thread-local
// error message, and launch checking.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdint>
#include "../../include/bi_abi.h"
#include "bi_math.cuh"

namespace bi {

// Defined in abi.cu. Records `msg` for bi_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);

// Defined in abi.cu: counts kernel launches of the library (read back by bi_launch_count()).
void count_launch();

inline int check_launch(const char* what) {
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(BI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return BI_OK;
}

// A runtime call other than a launch failed. Its error also stays in the slot that check_launch() reads, where the next
// launch would report it as its own: taken out here.
inline int fail_cuda(const char* what, cudaError_t e) {
    cudaGetLastError();
    return fail(BI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Defined in abi.cu: whether a kernel is launched with programmatic dependent launch; `peers`: it waits for or signals
// other ranks.
bool pdl_enabled(bool peers = false);

// Launch `kernel` so that it may begin (block scheduling, barrier and tensor-memory set-up) while the kernel before it
// on the stream is still draining; the kernel itself waits (ptx::grid_dep_wait) before it reads what earlier kernels wrote or
// writes anything. (A weight that its caller vouches for is read before that.)
// Every kernel launched through here MUST execute ptx::grid_dep_wait() in every CTA: completion of this kernel then
// implies completion of everything before it, which is what the kernel after it relies on.
// When the kernel after this one may begin is this kernel's to say (ptx::grid_dep_launch): matmuls say so when their last loads
// or MMAs are on their way, most others behind their own wait -- CTAs that sit resident from the start take room from
// them. A kernel that says nothing lets the next one in when its last CTAs leave.
// Kernels of several CTAs an SM need an even spread of them (spread_smem below) or are launched plainly.
template <typename... KArgs, typename... Args>
inline void launch_kernel(bool overlapped, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlapped ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);     // errors are picked up by check_launch()
}
template <typename... KArgs, typename... Args>
inline void launch_overlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    launch_kernel(pdl_enabled(), kernel, grid, block, smem, st, static_cast<Args&&>(args)...);
}
// The same for kernels that take part in a handshake with other ranks where `peers` is set.
template <typename... KArgs, typename... Args>
inline void launch_overlapped_unless(bool peers, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    launch_kernel(pdl_enabled(peers), kernel, grid, block, smem, st, static_cast<Args&&>(args)...);
}

inline bool aligned(const void* p, size_t n) { return (reinterpret_cast<uintptr_t>(p) % n) == 0; }

inline size_t dtype_size(int dtype) { return dtype == BI_F32 ? 4 : 2; }

inline bool dtype_ok(int dtype) { return dtype == BI_F32 || dtype == BI_F16 || dtype == BI_BF16; }

// Streaming multiprocessors of the current device (cached per device ordinal). Launch shapes are
// sized from it; no arithmetic depends on it.
inline int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!cached[dev]) cudaDeviceGetAttribute(&cached[dev], cudaDevAttrMultiProcessorCount, dev);
    return cached[dev] > 0 ? cached[dev] : 148;
}

// An SM's shared memory, of which every CTA takes 1 KB besides its own, and what a CTA may have.
constexpr size_t SM_SMEM = 228 << 10, CTA_SMEM = 227 << 10;

// The dynamic shared memory that a launch of KERNEL may ask for; the opt-in to it is made once per device. 0: refused.
template <auto KERNEL> size_t opt_in_smem() {
    static std::atomic<int> cached[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    int most = cached[dev].load(std::memory_order_relaxed);
    if (!most) {
        cudaFuncAttributes a;
        cudaError_t e = cudaFuncGetAttributes(&a, KERNEL);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, most = (int)(CTA_SMEM - a.sharedSizeBytes));
        if (e != cudaSuccess) { cudaGetLastError(); return 0; }                // not the next launch's error
        cached[dev].store(most, std::memory_order_relaxed);
    }
    return (size_t)most;
}

// CTAs of KERNEL that an SM holds, which is always launched with the same threads and shared memory; asked once per device.
template <auto KERNEL> int resident_ctas(int threads, size_t smem) {
    static std::atomic<int> cached[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    int n = cached[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, KERNEL, threads, smem) != cudaSuccess || n < 1) { cudaGetLastError(); return 32; }
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// CTAs that are let in beside a running kernel land where room comes free first, four on some SMs and none on others; a grid of
// less than a wave then takes as long as the fullest SM. A launch that asks for this much dynamic shared memory (`smem` is what
// KERNEL uses) leaves an SM no room for more CTAs than an even spread gives it.
template <auto KERNEL> size_t spread_smem(int64_t ctas, size_t smem) {
    const size_t fixed = CTA_SMEM - opt_in_smem<KERNEL>(), per_sm = (size_t)((ctas + sm_count() - 1) / sm_count());
    const size_t share = SM_SMEM / (per_sm + 1);                     // one CTA more would need more than all
    return share > fixed ? std::max(smem, (share - fixed + 127) / 128 * 128) : smem;
}

// Canonical constants of the arithmetic contract.
constexpr int GROUP_K = 256;  // K is folded in groups of this many elements, whatever M is

}  // namespace bi
