// The chunked LM-head loop (forward product, softmax cross entropy, input gradient) of the
// reference's production consumer (docs/mmq_bwd_optimization.md:502-524) and its element-wise part:
// per chunk of rows  logits = X W^T (bf16)  ->  loss += lse - logits[target],
// dlogits = (softmax - onehot) * scale (bf16, in place)  ->  dX = dlogits W.
//
// What bounds the element-wise part: HBM.  A chunk of 256 x 248320 logits is 127 MB, about the L2, so
// it is read twice (row statistics, then the gradient) and written once; the second pass walks the
// rows backwards because the last rows of the first are still in L2.  The separate passes of a
// framework (to fp32, log-softmax, gather, exp, scatter, scale, to bf16) move 13 times the bytes.
#include "../../include/tgo_mmq.h"

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace tgo {

int route_fail(int code, const char* msg);  // tgo_api.cu
int mmq_dx_f32(const void* dy, const void* packed_weight, void* dx, float* dx_f32, int64_t rows, int64_t out_features, int64_t in_features,
               int quant_type, void* workspace, int64_t workspace_bytes, void* stream);  // tgo_api.cu

constexpr int kXentThreads = 256;
constexpr int kXentMaxSplits = 16;   // parts of a row in the statistics pass

struct MaxSum {
    float m, s;   // maximum, sum of exp(x - m)
};
__device__ __forceinline__ MaxSum merge(MaxSum a, MaxSum b) {
    const float m = fmaxf(a.m, b.m);   // an empty part has m = -inf, s = 0
    return {m, (a.m == m ? a.s : a.s * expf(a.m - m)) + (b.m == m ? b.s : b.s * expf(b.m - m))};
}

// Elements of a row as 16-byte vectors: the first `head` ones and those after the last vector are
// taken one by one (rows of an odd vocabulary start at any 2-byte boundary).
struct RowVecs {
    int head;
    long long nvec, tail0;
};
__device__ __forceinline__ RowVecs row_vecs(long long row, long long vocab) {
    RowVecs r;
    r.head = static_cast<int>((8 - (row * vocab) % 8) % 8);
    if (r.head > vocab) r.head = static_cast<int>(vocab);
    r.nvec = (vocab - r.head) / 8;
    r.tail0 = r.head + r.nvec * 8;
    return r;
}

__global__ void __launch_bounds__(kXentThreads) xent_stats_kernel(const __nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets,
                                                                  long long vocab, MaxSum* __restrict__ part, float* __restrict__ target_logit) {
    const long long row = blockIdx.y;
    const __nv_bfloat16* x = logits + row * vocab;
    const RowVecs r = row_vecs(row, vocab);
    MaxSum acc = {-INFINITY, 0.0f};
    auto take = [&](float v) { acc = merge(acc, {v, v == -INFINITY ? 0.0f : 1.0f}); };
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            const long long t = targets[row];
            // an id outside the vocabulary has no probability: the loss says so
            target_logit[row] = t >= 0 && t < vocab ? __bfloat162float(x[t]) : NAN;
        }
        if (threadIdx.x < r.head) take(__bfloat162float(x[threadIdx.x]));
        if (threadIdx.x < vocab - r.tail0) take(__bfloat162float(x[r.tail0 + threadIdx.x]));
    }
    const uint4* v = reinterpret_cast<const uint4*>(x + r.head);
    for (long long i = blockIdx.x * static_cast<long long>(kXentThreads) + threadIdx.x; i < r.nvec; i += gridDim.x * static_cast<long long>(kXentThreads)) {
        const uint4 q = v[i];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        float f[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            f[2 * j] = __uint_as_float(w[j] << 16);
            f[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
        }
        float m = f[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) m = fmaxf(m, f[j]);
        if (m > acc.m) {
            acc.s *= expf(acc.m - m);   // acc.m = -inf at first: 0 * 0
            acc.m = m;
        }
        // nothing but -inf so far (they add exp(-inf) = 0) and NaN (which no maximum shows, but the sum does)
        const float base = acc.m == -INFINITY ? 0.0f : acc.m;
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s += expf(f[j] - base);
        acc.s += s;
    }
    __shared__ MaxSum warp_part[kXentThreads / 32];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const MaxSum o = {__shfl_xor_sync(0xFFFFFFFFu, acc.m, d), __shfl_xor_sync(0xFFFFFFFFu, acc.s, d)};
        acc = merge(acc, o);
    }
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kXentThreads / 32; ++w) acc = merge(acc, warp_part[w]);
        part[row * gridDim.x + blockIdx.x] = acc;
    }
}

__global__ void __launch_bounds__(kXentThreads) xent_grad_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets,
                                                                 long long vocab, const MaxSum* __restrict__ part, const float* __restrict__ target_logit,
                                                                 float scale, float* __restrict__ row_loss) {
    const long long row = gridDim.y - 1 - blockIdx.y;
    __nv_bfloat16* x = logits + row * vocab;
    const RowVecs r = row_vecs(row, vocab);
    MaxSum all = part[row * gridDim.x];
    for (int i = 1; i < static_cast<int>(gridDim.x); ++i) all = merge(all, part[row * gridDim.x + i]);
    const float lse = all.m + logf(all.s);
    const long long target = targets[row];
    auto grad = [&](float v, long long col) { return (expf(v - lse) - (col == target ? 1.0f : 0.0f)) * scale; };
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) row_loss[row] = lse - target_logit[row];
        if (threadIdx.x < r.head) x[threadIdx.x] = __float2bfloat16(grad(__bfloat162float(x[threadIdx.x]), threadIdx.x));
        if (threadIdx.x < vocab - r.tail0) {
            const long long c = r.tail0 + threadIdx.x;
            x[c] = __float2bfloat16(grad(__bfloat162float(x[c]), c));
        }
    }
    uint4* v = reinterpret_cast<uint4*>(x + r.head);
    for (long long i = blockIdx.x * static_cast<long long>(kXentThreads) + threadIdx.x; i < r.nvec; i += gridDim.x * static_cast<long long>(kXentThreads)) {
        const uint4 q = v[i];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        const long long col = r.head + i * 8;
        float p[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            p[2 * j] = expf(__uint_as_float(w[j] << 16) - lse) * scale;
            p[2 * j + 1] = expf(__uint_as_float(w[j] & 0xFFFF0000u) - lse) * scale;
        }
        if (static_cast<unsigned long long>(target - col) < 8ull) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (target == col + j) p[j] = grad(__uint_as_float(j & 1 ? w[j >> 1] & 0xFFFF0000u : w[j >> 1] << 16), col + j);
        }
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(p[2 * j], p[2 * j + 1]);
            o[j] = *reinterpret_cast<const uint32_t*>(&b);
        }
        v[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// loss = sum of the rows' losses, one block, fixed order
__global__ void __launch_bounds__(256) sum_rows_kernel(const float* __restrict__ row_loss, long long rows, float* __restrict__ loss) {
    float s = 0.0f;
    for (long long r = threadIdx.x; r < rows; r += 256) s += row_loss[r];
    __shared__ float warp_sum[8];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, d);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s += warp_sum[w];
        *loss = s;
    }
}

// parts of a row: enough blocks for the SMs when there are few rows
static int xent_splits(int64_t rows) {
    const int64_t s = (148 * 8 + rows - 1) / rows;
    return static_cast<int>(s > kXentMaxSplits ? kXentMaxSplits : s);
}
static int64_t up256(int64_t n) { return (n + 255) & ~static_cast<int64_t>(255); }

// workspace: logits of one chunk, row losses, the chunk's target logits and statistics, split-reduction sums
struct HeadSpace {
    int64_t row_loss, target_logit, part, dx_ws, total;
};
static HeadSpace head_space(int64_t rows, int64_t vocab, int64_t k, int qt, int64_t chunk) {
    HeadSpace s;
    s.row_loss = up256(chunk * vocab * 2);
    s.target_logit = s.row_loss + up256(rows * 4);
    s.part = s.target_logit + up256(chunk * 4);
    s.dx_ws = s.part + up256(chunk * kXentMaxSplits * static_cast<int64_t>(sizeof(MaxSum)));
    int64_t dx = tgo_mmq_dx_workspace_bytes(chunk, vocab, k, qt);
    const int64_t last = rows % chunk;
    if (last != 0) {
        const int64_t b = tgo_mmq_dx_workspace_bytes(last, vocab, k, qt);
        if (b > dx) dx = b;
    }
    s.total = s.dx_ws + dx;
    return s;
}

}  // namespace tgo

using namespace tgo;

extern "C" {

int64_t tgo_lm_head_loss_workspace_bytes(int64_t rows, int64_t vocab, int64_t in_features, int quant_type, int64_t chunk_rows) {
    if (rows <= 0 || vocab <= 0 || in_features <= 0 || chunk_rows <= 0 || tgo_block_bytes(quant_type) < 0) return -1;
    return head_space(rows, vocab, in_features, quant_type, chunk_rows < rows ? chunk_rows : rows).total;
}

int tgo_lm_head_loss_f32(const void* hidden, const void* packed_weight, const int64_t* targets, int64_t rows, int64_t vocab,
                         int64_t in_features, int quant_type, int64_t chunk_rows, float grad_scale, float* loss, void* d_hidden,
                         float* d_hidden_f32, void* workspace, int64_t workspace_bytes, void* stream) {
    if (targets == nullptr || loss == nullptr || workspace == nullptr) return route_fail(TGO_E_ARG, "null pointer");
    if (chunk_rows <= 0) return route_fail(TGO_E_ARG, "chunk_rows must be positive");
    if (rows <= 0) return route_fail(TGO_E_ARG, "zero-row inputs are not supported");
    const int64_t chunk = chunk_rows < rows ? chunk_rows : rows;
    const int64_t need = tgo_lm_head_loss_workspace_bytes(rows, vocab, in_features, quant_type, chunk);
    if (need < 0) return route_fail(TGO_E_ARG, "unsupported quant_type or sizes");
    if (workspace_bytes < need) return route_fail(TGO_E_WORKSPACE, "workspace is smaller than tgo_lm_head_loss_workspace_bytes");
    const HeadSpace sp = head_space(rows, vocab, in_features, quant_type, chunk);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    __nv_bfloat16* logits = reinterpret_cast<__nv_bfloat16*>(ws);
    float* row_loss = reinterpret_cast<float*>(ws + sp.row_loss);
    float* target_logit = reinterpret_cast<float*>(ws + sp.target_logit);
    MaxSum* part = reinterpret_cast<MaxSum*>(ws + sp.part);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int64_t b = 0; b < rows; b += chunk) {
        const int64_t n = rows - b < chunk ? rows - b : chunk;
        const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(hidden) + b * in_features;
        int rc = tgo_mmq_fwd(x, packed_weight, logits, n, vocab, in_features, quant_type, stream);
        if (rc != TGO_OK) return rc;
        const int splits = xent_splits(n);
        constexpr int64_t kRows = 65528;   // most rows of a grid, a multiple of 8: every part starts 16-byte aligned
        for (int64_t r = 0; r < n; r += kRows) {
            const int64_t m = n - r < kRows ? n - r : kRows;
            const dim3 grid(splits, static_cast<unsigned>(m));
            xent_stats_kernel<<<grid, kXentThreads, 0, st>>>(logits + r * vocab, targets + b + r, vocab, part + r * splits, target_logit + r);
            xent_grad_kernel<<<grid, kXentThreads, 0, st>>>(logits + r * vocab, targets + b + r, vocab, part + r * splits, target_logit + r,
                                                            grad_scale, row_loss + b + r);
        }
        if (cudaGetLastError() != cudaSuccess) return route_fail(TGO_E_CUDA, "cross-entropy kernel launch failed");
        rc = mmq_dx_f32(logits, packed_weight, static_cast<__nv_bfloat16*>(d_hidden) + b * in_features,
                        d_hidden_f32 != nullptr ? d_hidden_f32 + b * in_features : nullptr, n, vocab, in_features, quant_type, ws + sp.dx_ws,
                        sp.total - sp.dx_ws, stream);
        if (rc != TGO_OK) return rc;
    }
    sum_rows_kernel<<<1, 256, 0, st>>>(row_loss, rows, loss);
    return cudaGetLastError() == cudaSuccess ? TGO_OK : route_fail(TGO_E_CUDA, "sum_rows_kernel launch failed");
}

int tgo_lm_head_loss(const void* hidden, const void* packed_weight, const int64_t* targets, int64_t rows, int64_t vocab,
                     int64_t in_features, int quant_type, int64_t chunk_rows, float grad_scale, float* loss, void* d_hidden,
                     void* workspace, int64_t workspace_bytes, void* stream) {
    return tgo_lm_head_loss_f32(hidden, packed_weight, targets, rows, vocab, in_features, quant_type, chunk_rows, grad_scale, loss, d_hidden,
                                nullptr, workspace, workspace_bytes, stream);
}

}  // extern "C"
