// Host-side launch interface between the C-ABI layer (tgo_api.cu) and the per-quant-type
// instantiations of the few-token kernel (mmq_small_inst.cu, compiled once per type).
#pragma once

#include "mmq_small.cuh"

namespace tgo {

constexpr int kSmallSmemLimit = 232448;   // 227 KB opt-in limit per CTA

// launch_small_<QT>: launches mmq_small_kernel<QT, nt> (8 * nt tokens per tile) with `grid`
// persistent CTAs of kw * rw warps.  Returns a cudaError_t.
// small_smem_<QT>: dynamic shared memory of such a launch.
#define TGO_DECLARE_SMALL(QT)                                                                       \
    int launch_small_##QT(int nt, const SmallArgs& args, int grid, int smem, cudaStream_t stream); \
    int small_smem_##QT(int nkb, int nt, int kw, int rw, int stages, int groups);
TGO_DECLARE_SMALL(11)
TGO_DECLARE_SMALL(12)
TGO_DECLARE_SMALL(13)
TGO_DECLARE_SMALL(14)
TGO_DECLARE_SMALL(22)
#undef TGO_DECLARE_SMALL

}  // namespace tgo
