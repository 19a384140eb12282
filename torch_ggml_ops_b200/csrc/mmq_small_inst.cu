// One translation unit per quant type (compile with -DTGO_QT=<ggml type id>): the few-token forward
// kernel for 8, 16, 24 and 32 tokens per tile, and its launch function.
#include <atomic>

#include "mmq_small_launch.h"

#ifndef TGO_QT
#error "compile with -DTGO_QT=<11|12|13|14|22>"
#endif

namespace tgo {

template <int NT>
static int launch_nt(const SmallArgs& args, int grid, int smem, cudaStream_t stream) {
    // relaxed atomics: threads that race on a device's first call set the same attribute and flag
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(mmq_small_kernel<TGO_QT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmemLimit);
        if (e != cudaSuccess) return static_cast<int>(e);
        if (dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    mmq_small_kernel<TGO_QT, NT><<<grid, args.kw * args.rw * 32, smem, stream>>>(args);
    return static_cast<int>(cudaGetLastError());
}

#define TGO_CAT2(a, b) a##b
#define TGO_CAT(a, b) TGO_CAT2(a, b)

int TGO_CAT(launch_small_, TGO_QT)(int nt, const SmallArgs& args, int grid, int smem, cudaStream_t stream) {
    switch (nt) {
        case 1: return launch_nt<1>(args, grid, smem, stream);
        case 2: return launch_nt<2>(args, grid, smem, stream);
        case 3: return launch_nt<3>(args, grid, smem, stream);
        default: return launch_nt<4>(args, grid, smem, stream);
    }
}

int TGO_CAT(small_smem_, TGO_QT)(int nkb, int nt, int kw, int rw, int stages, int groups) {
    return small_smem_bytes<TGO_QT>(nkb, nt, kw, rw, stages, groups);
}

}  // namespace tgo
