// Shared host/device helpers of the CUDA library: status handling, activation functions, launch counting.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <atomic>

#include "../../include/dlp_cuda.h"

namespace dlp {

// ---- host side: per-thread error message, launch counter --------------------------------------
void set_error(const std::string &msg);
dlp_status fail(dlp_status st, const std::string &msg);
dlp_status check_cuda(cudaError_t e, const char *what);
extern std::atomic<uint64_t> g_launches;
inline void count_launch(int n = 1) { g_launches.fetch_add(uint64_t(n), std::memory_order_relaxed); }
int sm_count();

#define DLP_REQUIRE(cond, msg)                                                             \
    do {                                                                                   \
        if(!(cond)) return ::dlp::fail(DLP_INVALID_ARGUMENT, std::string("Failed " #cond ": ") + (msg)); \
    } while(0)

#define DLP_CUDA_OK(expr)                                                                  \
    do {                                                                                   \
        dlp_status st__ = ::dlp::check_cuda((expr), #expr);                                \
        if(st__ != DLP_OK) return st__;                                                    \
    } while(0)

// expr: a launch_pdl call
#define DLP_LAUNCH_PDL(expr, name)                                                         \
    do {                                                                                   \
        dlp_status st__ = ::dlp::check_cuda((expr), name);                                 \
        if(st__ != DLP_OK) return st__;                                                    \
        ::dlp::count_launch();                                                             \
    } while(0)

#define DLP_LAUNCH_OK(name)                                                                \
    do {                                                                                   \
        ::dlp::count_launch();                                                             \
        dlp_status st__ = ::dlp::check_cuda(cudaPeekAtLastError(), name);                  \
        if(st__ != DLP_OK) return st__;                                                    \
    } while(0)

// Launch of a kernel of the path.  `early`: it may start while the kernel before it on the stream is still running
// (programmatic dependent launch): its blocks are set up -- and wait in pdl_wait() -- under the other's last blocks instead of
// after them.  The waiting is the kernel's own: every kernel launched this way calls pdl_wait() in each thread before its first
// access to global memory (but for the index tables of a plan, which no kernel writes), and before its first wait for another warp: those waits are limited in time, and the kernel before
// may take longer than the limit.  A kernel or copy of somebody else's before or after it is ordered in full as ever.
// For launches whose blocks all fit on the GPU at once (one_wave): there the set-up is a good part of the time (InnerProduct
// 2048 -> 1000 on one row 24.6 -> 21.3 us, on 256 rows with its packing 38.9 -> 33.3 us).  Longer launches lose more than
// the set-up they hide: an SM that takes its first block of the new kernel while the old one still runs keeps the old one's
// split of L1 and shared memory (depthwise 3x3 144x56x56 + 1x1 at batch 128 175 -> 196 us, ResNet-50 at 256 14.0 -> 15.0 ms).
template<typename... P, typename... A>
inline cudaError_t launch_pdl(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A &...args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Blocks of a plain kernel (threads each) that are all resident at once as far as threads go; where registers or shared memory allow fewer
// (global pooling's tiles, the banded depthwise kernel) it is a round or two more.  Captured chains of one layer, never early -> early
// (us): depthwise 3x3 144x56x56 at 1, 4 and 8 images 4.0 -> 3.6, 5.9 -> 5.5, 9.1 -> 8.7, 960x7x7 at 32 8.2 -> 7.9; beyond the line no
// difference to speak of (96x112x112 and 960x7x7 at 128: within 0.2), and behind other kernels a loss (above).
inline bool one_wave(long long blocks, int threads) { return blocks * threads <= (long long)sm_count() * 2048; }
// Work items of a persistent tensor-core kernel that are few enough for the set-up to matter.  Captured chains of one layer, never
// early -> early (us): 3x3 64 -> 64 on 56x56 at batch 4, 16 and 21 (112, 448 and 588 items) 14.2 -> 13.1, 36.8 -> 34.6, 36.9 -> 35.5;
// 3x3 128 -> 128 on 28x28 at 16 27.3 -> 25.8; 1x1 64 -> 256 on 56x56 with residual at 4 and 11 13.6 -> 12.6, 19.2 -> 18.2; 1x1 256 ->
// 1024 on 14x14 with residual at 16 and 32 18.9 -> 17.5, 25.5 -> 24.7, but at 48 (592 items) 34.8 -> 36.5.  Further on a chain of one
// layer would still gain up to 2 us (batch 22 to 48 of the first), a network of different layers loses (above).
inline bool few_items(long long items) { return items <= 4ll * sm_count(); }

// ---- device side ---------------------------------------------------------------------------------
// Activation definitions shared by every epilogue; they follow the reference's device macros
// (src/kernels/defs.h:27-49) and its CPU versions (include/dlprim/cpu/cpu_ops.hpp:16-53).
// tanhf/expf are the accurate library forms, not the .approx instructions.
__device__ __forceinline__ float apply_act(float v, int act)
{
    switch(act) {
    case DLP_ACT_RELU: return fmaxf(v, 0.0f);
    case DLP_ACT_TANH: return tanhf(v);
    case DLP_ACT_SIGMOID: return 1.0f / (1.0f + expf(-v));
    case DLP_ACT_RELU6: return fminf(fmaxf(v, 0.0f), 6.0f);
    default: return v;
    }
}

// Waits until the kernels this one depends on are complete and their writes visible, then lets the next kernel's blocks be set
// up.  In that order: a kernel never starts before the one two places ahead of it is complete.
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Load of what a kernel before this one may have written.  A kernel that starts early is resident while that one writes, so these
// are not the read-only loads (__ldg, pointers to const with __restrict__), which are for memory that nobody writes while the kernel
// lives and which nothing holds behind pdl_wait().  Stores through pointers that may overlap hold plain loads back: loops with many
// of them ask for what they read before they store.
template<typename T> __device__ __forceinline__ T ld_plain(const T *p) { return *p; }

template<typename T> __host__ __device__ inline T ceil_div(T a, T b) { return (a + b - 1) / b; }
template<typename T> __host__ __device__ inline T round_up(T a, T b) { return ceil_div(a, b) * b; }

// Device address of the per-device status word written by kernels whose bounded waits gave up
// (0 = healthy).  Resolved once per device; never allocates.
int *device_status_word();

} // namespace dlp
