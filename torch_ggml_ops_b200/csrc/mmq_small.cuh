// The forward product for few tokens per weight row (decode batches, sparsely hit experts): a
// memory-bound kernel beside the tile GEMM of mmq_gemm.cuh.
//
//   Y[t, n] = sum_k X[t, k] * W[n, k]      (reference: csrc/mmq_core.cuh:211-267, 450-514, 573-635)
//
// What bounds it: every packed byte of the weight is used once, so the floor is the copy rate of
// HBM; at that rate an SM has to unpack some 28 (Q6_K) to 80 (Q4_K) weights per clock, three to
// four times what the GEMM's decode warps reach, and most calls are so small that latency counts.
// Hence:
//
// * The contraction runs on mma.sync m16n8k16 (16 weight rows x 8 tokens): the operand that the
//   bits are unpacked into is a register fragment, so a decoded weight never goes through shared
//   memory, there is no descriptor, barrier or TMEM hand-off per step, and a warp works alone.
// * Scales stay out of the weights.  The fragments hold 128 + q (exact in bf16: the byte q under the
//   exponent byte 0x43, one byte permute per two weights), and the scale of a 32- or 16-weight group
//   multiplies the fp32 partial sum.  Offsets (the 128, the types' own, the minima of Q4_K / Q5_K)
//   are two more mma per block: scales and minima, exact in bf16, against the group sums of x, split
//   into two bf16 parts (16 bits).  No weight is rounded to bf16 at all.
//   IQ2_S, whose mma cover two scale groups, holds 3 * magnitude * scale, rounded once to bf16 as the
//   GEMM's weights are, and the block's fp16 scale multiplies the fp32 partial sum.
// * The k order inside a 32-weight group is permuted so that a thread's fragment elements are the
//   bytes of the words it reads; the activations are laid out once per token tile in the same
//   order (shared memory, one 16-byte load per lane, two mma and eight tokens).
// * A CTA is kw x rw warps: kw slices of the reduction times rw tiles of 16 weight rows.  Every
//   warp streams its own blocks with cp.async (16 rows x one block per stage, stages deep) and
//   needs no other warp until the partial sums of the kw slices meet in shared memory.
// * Persistent CTAs take contiguous ranges of the (token tile, weight set, row tile) units, so the
//   activation fragments are rebuilt only where the token tile changes.  Grouped calls find their
//   token tiles by a prefix sum over the groups in every CTA: no tile list, no second launch.
// * The bias and the group sums take an infinite activation or block scale to inf - inf, and leave
//   fp32's range before the product does (from |x| of some 1e36, 1e26 with the largest scales).  Both
//   show as a sum that is not finite, and such sums alone are computed again from decoded weights, as
//   the GEMM does; nothing of that is in the loop over the blocks.
#pragma once

#include "gguf_decode.cuh"
#include "ptx.cuh"

namespace tgo {

constexpr int kSmallMaxSets = 4;
constexpr int kSmallMaxGroups = 1024;   // groups whose prefix sum a CTA keeps in shared memory
constexpr int kSmallWarps = 16;         // most warps of a CTA

struct SmallArgs {
    const uint8_t* wgt[kSmallMaxSets];
    __nv_bfloat16* out[kSmallMaxSets];
    const __nv_bfloat16* act;
    const int64_t* experts;              // null: dense
    const int32_t* offsets;
    __nv_bfloat16* const* out_rows;      // per-row destinations of one weight set, or null
    const uint64_t* iq2s_grid;
    int* tile_count;                     // grouped: receives the number of token tiles, as the GEMM's tile list does
    long long wgt_bytes;                 // bytes of one packed tensor (all experts)
    int rows, out_features, in_features;
    int nsets, groups, num_experts;
    int row_bytes;
    int kw, rw, stages;
};

// Layout of one warp stage: 16 block windows (see BlockFmt) of kPitch bytes, which puts the 8 rows x
// 4 lanes of a fragment load on different banks: 32-bit loads want a pitch of 4 (mod 8) words, the
// 64-bit loads of the aligned types 8 (mod 16; Q5_K's 44 words cost every fourth row a second pass,
// padding would cost a stage).
template <int QT> struct SmallFmt {
    using Fmt = BlockFmt<QT>;
    static constexpr bool kAffine = QT == QT_Q4_K || QT == QT_Q5_K;
    static constexpr bool kScaled16 = QT == QT_Q6_K || QT == QT_Q3_K;
    static constexpr int kPitch = QT == QT_Q4_K ? 160 : QT == QT_Q5_K ? 176 : Fmt::kSlot;
    static constexpr int kChunks = Fmt::kCopy / 16;            // 16-byte pieces of a window
    static constexpr int kStageBytes = 16 * kPitch;
    // k order inside a 32-weight group: thread t of a quad holds k = 8t + 4i + 0..3 (its two words
    // are neighbours) or k = 16i + 4t + 0..3 (16-weight scale groups), i = which of the two mma
    static constexpr bool kPairOrder = !kScaled16;
    static constexpr int kGridBytes = QT == QT_IQ2_S ? 8192 : 0;
    static constexpr float kBias = QT == QT_Q6_K ? 160.0f : QT == QT_Q3_K ? 132.0f : 128.0f;   // fragment minus quant
    // group-sum fragments per block and 8 tokens: sums of 8 groups in two bf16 parts fill one mma, of 16 groups two
    static constexpr int kSumBytes = kAffine ? 256 : kScaled16 ? 512 : 0;
};

// shared memory of a launch, in the order of the carve-up
template <int QT>
__host__ __device__ inline int small_frag_bytes(int nkb, int nt) {
    return nkb * nt * (8 * 512 + SmallFmt<QT>::kSumBytes);
}
template <int QT>
__host__ __device__ inline int small_smem_bytes(int nkb, int nt, int kw, int rw, int stages, int groups) {
    return small_frag_bytes<QT>(nkb, nt) + SmallFmt<QT>::kGridBytes + kw * rw * stages * SmallFmt<QT>::kStageBytes +
           (kw > 1 ? 2 * kw * rw * nt * 512 : 0) + groups * 12 + 256;
}

// d += a b;  d = a b
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// tot += (s0, s1 for the two rows) * acc
__device__ __forceinline__ void add_scaled(float (&tot)[4], float s0, float s1, const float (&acc)[4]) {
    const float2 u = __ffma2_rn(make_float2(s0, s0), make_float2(acc[0], acc[1]), make_float2(tot[0], tot[1]));
    const float2 v = __ffma2_rn(make_float2(s1, s1), make_float2(acc[2], acc[3]), make_float2(tot[2], tot[3]));
    tot[0] = u.x; tot[1] = u.y; tot[2] = v.x; tot[3] = v.y;
}
// 16 bytes global -> shared; bytes past `n` are filled with zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int n) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bar_named(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t hadd2_bf16(uint32_t a, uint32_t b) { return as_u32(__hadd2(as_bf162(a), as_bf162(b))); }
__device__ __forceinline__ uint32_t hmul2_bf16(uint32_t a, uint32_t b) { return as_u32(__hmul2(as_bf162(a), as_bf162(b))); }
// bytes 0, 1 (or 2, 3) of v under the exponent byte `top`: the bf16 pair 128 + byte for 0x43
__device__ __forceinline__ uint32_t bytes01(uint32_t v, uint32_t top) { return __byte_perm(v, top, 0x4140); }
__device__ __forceinline__ uint32_t bytes23(uint32_t v, uint32_t top) { return __byte_perm(v, top, 0x4342); }
constexpr uint32_t kTop128 = 0x43434343u, kMinus128 = 0xC300C300u, kMinus160 = 0xC320C320u;

// byte b of v as the float 2^15 + byte
__device__ __forceinline__ float byte_plus_32768(uint32_t v, int b) {
    return __uint_as_float(__byte_perm(v, 0x47000000u, 0x7604u + 0x10u * b));
}

// 32-bit word `off` bytes (a multiple of 4) after a block start whose address rounded down to 4 is
// `base`; `sh` = 0 or 16 bits of misalignment
__device__ __forceinline__ uint32_t ld_word_at(uint32_t base, uint32_t off, uint32_t sh) {
    return __funnelshift_r(lds32(base + off), lds32(base + off + 4), sh);
}

// One block (256 weights) of 16 rows against all tokens of the tile, added to `tot`.
//   p0, p1: shared addresses of this thread's two rows' blocks (rows lane / 4 and lane / 4 + 8)
//   frag: this block's x fragments plus lane * 16;  sums: its group-sum fragments plus lane * 8
template <int QT, int NT> struct SmallBlock;

template <int QT, int NT> struct SmallAffine {
    __device__ static __forceinline__ void run(uint32_t p0, uint32_t p1, uint32_t frag, uint32_t sums, uint32_t, int lane, float (&tot)[NT][4]) {
        const int t = lane & 3;
        const uint4 h0 = lds128(p0), h1 = lds128(p1);
        const float d0 = half_bits_to_float(h0.x & 0xFFFFu), d1 = half_bits_to_float(h1.x & 0xFFFFu);
        const uint32_t sc0[2] = {h0.y & 0x3F3F3F3Fu, (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u)};
        const uint32_t sc1[2] = {h1.y & 0x3F3F3F3Fu, (h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u)};
        {   // offsets of all groups: dmin * minimum + 128 d * scale, against the group sums.  k slots of thread
            // t are groups 4 (t & 1) + 0..3 of the sums' high (t < 2) or low part.
            const bool odd = (t & 1) != 0;
            const uint32_t m0 = odd ? ((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u) : h0.z & 0x3F3F3F3Fu;
            const uint32_t m1 = odd ? ((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u) : h1.z & 0x3F3F3F3Fu;
            const uint32_t c0 = odd ? sc0[1] : sc0[0], c1 = odd ? sc1[1] : sc1[0];
            const uint32_t a[4] = {hadd2_bf16(bytes01(m0, kTop128), kMinus128), hadd2_bf16(bytes01(m1, kTop128), kMinus128),
                                   hadd2_bf16(bytes23(m0, kTop128), kMinus128), hadd2_bf16(bytes23(m1, kTop128), kMinus128)};
            const uint32_t b[4] = {hadd2_bf16(bytes01(c0, kTop128), kMinus128), hadd2_bf16(bytes01(c1, kTop128), kMinus128),
                                   hadd2_bf16(bytes23(c0, kTop128), kMinus128), hadd2_bf16(bytes23(c1, kTop128), kMinus128)};
            const float n0 = -half_bits_to_float(h0.x >> 16), n1 = -half_bits_to_float(h1.x >> 16);
            const float o0 = -128.0f * d0, o1 = -128.0f * d1;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 x = lds64(sums + nt * 256);
                float acc[4];
                mma_bf16_first(acc, a, x.x, x.y);
                add_scaled(tot[nt], n0, n1, acc);
                mma_bf16_first(acc, b, x.x, x.y);
                add_scaled(tot[nt], o0, o1, acc);
            }
        }
        constexpr uint32_t kQs = QT == QT_Q5_K ? 48 : 16;
        uint2 q50 = make_uint2(0, 0), q51 = make_uint2(0, 0);   // Q5_K: bit g of byte b is the fifth bit of weight b of group g
        if (QT == QT_Q5_K) {
            q50 = lds64(p0 + 16 + 8 * t);
            q51 = lds64(p1 + 16 + 8 * t);
        }
        // the bias 2^23 of a byte as a float comes off in the product: exact, d * scale fits fp32
        const float e0 = -8388608.0f * d0, e1 = -8388608.0f * d1;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint2 q0 = lds64(p0 + kQs + 32 * s + 8 * t), q1 = lds64(p1 + kQs + 32 * s + 8 * t);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = 2 * s + h;
                uint32_t v[4] = {(q0.x >> (4 * h)) & 0x0F0F0F0Fu, (q1.x >> (4 * h)) & 0x0F0F0F0Fu,
                                 (q0.y >> (4 * h)) & 0x0F0F0F0Fu, (q1.y >> (4 * h)) & 0x0F0F0F0Fu};
                if (QT == QT_Q5_K) {
                    const uint32_t w[4] = {q50.x, q51.x, q50.y, q51.y};
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] |= (g <= 4 ? w[i] << (4 - g) : w[i] >> (g - 4)) & 0x10101010u;
                }
                const uint32_t a[4] = {bytes01(v[0], kTop128), bytes01(v[1], kTop128), bytes23(v[0], kTop128), bytes23(v[1], kTop128)};
                const uint32_t b[4] = {bytes01(v[2], kTop128), bytes01(v[3], kTop128), bytes23(v[2], kTop128), bytes23(v[3], kTop128)};
                const float ds0 = fmaf(d0, byte_to_biased_float(sc0[g >> 2], g & 3), e0);
                const float ds1 = fmaf(d1, byte_to_biased_float(sc1[g >> 2], g & 3), e1);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint4 x = lds128(frag + (g * NT + nt) * 512);
                    float acc[4];
                    mma_bf16_first(acc, a, x.x, x.y);
                    mma_bf16(acc, b, x.z, x.w);
                    add_scaled(tot[nt], ds0, ds1, acc);
                }
            }
        }
    }
};
template <int NT> struct SmallBlock<QT_Q4_K, NT> : SmallAffine<QT_Q4_K, NT> {};
template <int NT> struct SmallBlock<QT_Q5_K, NT> : SmallAffine<QT_Q5_K, NT> {};

// Q6_K and Q3_K: one scale per 16 weights, i.e. per mma.
template <int QT, int NT> struct SmallScaled16 {
    __device__ static __forceinline__ void run(uint32_t p0, uint32_t p1, uint32_t frag, uint32_t sums, uint32_t, int lane, float (&tot)[NT][4]) {
        const int t = lane & 3;
        const uint32_t b0 = p0 & ~3u, b1 = p1 & ~3u, sh0 = (p0 & 2u) * 8u, sh1 = (p1 & 2u) * 8u;
        constexpr bool k6 = QT == QT_Q6_K;
        constexpr uint32_t kD = k6 ? 208 : 108;
        float d[2] = {half_bits_to_float(lds16(p0 + kD)), half_bits_to_float(lds16(p1 + kD))};
        // scales as unsigned bytes (Q6_K: + 128, Q3_K: + 32); their bias and the 2^15 of a byte under
        // that exponent come off in the product.  All exact: the bias times d has at most 22 bits.
        uint32_t sc[2][4];
        float e[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t b = r == 0 ? b0 : b1, sh = r == 0 ? sh0 : sh1;
            if (k6) {
#pragma unroll
                for (int j = 0; j < 4; ++j) sc[r][j] = ld_word_at(b, 192 + 4 * j, sh) ^ 0x80808080u;
                e[r] = -(32768.0f + 128.0f) * d[r];
            } else {
                const uint32_t s0 = ld_word_at(b, 96, sh), s1 = ld_word_at(b, 100, sh), s2 = ld_word_at(b, 104, sh);
                sc[r][0] = (s0 & 0x0F0F0F0Fu) | ((s2 << 4) & 0x30303030u);
                sc[r][1] = (s1 & 0x0F0F0F0Fu) | ((s2 << 2) & 0x30303030u);
                sc[r][2] = ((s0 >> 4) & 0x0F0F0F0Fu) | (s2 & 0x30303030u);
                sc[r][3] = ((s1 >> 4) & 0x0F0F0F0Fu) | ((s2 >> 2) & 0x30303030u);
                e[r] = -(32768.0f + 32.0f) * d[r];
            }
        }
        {   // offsets of all groups against the group sums: k slots of thread t are scales 4 t + 0..3, high
            // parts of the sums in the first mma, low parts in the second
            uint32_t a[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t w = t < 2 ? (t == 0 ? sc[r][0] : sc[r][1]) : (t == 2 ? sc[r][2] : sc[r][3]);
                // Q6_K: bytes hold s + 128; s = (128 + low 7 bits) - 128 if the top bit is set, - 256 if not
                const uint32_t lo = k6 ? w & 0x7F7F7F7Fu : w, up = k6 ? ~w & 0x80808080u : 0u;
                const uint32_t m01 = k6 ? __byte_perm(up, 0xC3C3C3C3u, 0x4140) : kMinus160;
                const uint32_t m23 = k6 ? __byte_perm(up, 0xC3C3C3C3u, 0x4342) : kMinus160;
                a[r] = hadd2_bf16(bytes01(lo, kTop128), m01);
                a[2 + r] = hadd2_bf16(bytes23(lo, kTop128), m23);
            }
            const float o0 = -SmallFmt<QT>::kBias * d[0], o1 = -SmallFmt<QT>::kBias * d[1];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 x = lds64(sums + nt * 512), y = lds64(sums + nt * 512 + 256);
                float acc[4];
                mma_bf16_first(acc, a, x.x, x.y);
                mma_bf16(acc, a, y.x, y.y);
                add_scaled(tot[nt], o0, o1, acc);
            }
        }
        // adds the two mma of 32-weight group g, whose byte-sized quants are v[row][i]
        auto group = [&](int g, const uint32_t (&v)[2][2]) {
            uint32_t a[2][4];
            float ds[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int k = 2 * g + i;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    a[i][r] = bytes01(v[r][i], kTop128);
                    a[i][2 + r] = bytes23(v[r][i], kTop128);
                    ds[i][r] = fmaf(d[r], byte_plus_32768(sc[r][k >> 2], k & 3), e[r]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 x = lds128(frag + (g * NT + nt) * 512);
                float acc[4];
                mma_bf16_first(acc, a[0], x.x, x.y);
                add_scaled(tot[nt], ds[0][0], ds[0][1], acc);
                mma_bf16_first(acc, a[1], x.z, x.w);
                add_scaled(tot[nt], ds[1][0], ds[1][1], acc);
            }
        };
        uint32_t hm[2][2];   // Q3_K: bit g of byte b is the third bit of weight b of group g
        if (!k6) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                hm[0][i] = ld_word_at(b0, 16 * i + 4 * t, sh0);
                hm[1][i] = ld_word_at(b1, 16 * i + 4 * t, sh1);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t q[2][2];   // [row][i] Q6_K: high bit pairs, Q3_K: low bit pairs of the half's four groups
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                q[0][i] = ld_word_at(b0, (k6 ? 128 : 32) + c * 32 + 16 * i + 4 * t, sh0);
                q[1][i] = ld_word_at(b1, (k6 ? 128 : 32) + c * 32 + 16 * i + 4 * t, sh1);
            }
            if (k6) {
#pragma unroll
                for (int k1 = 0; k1 < 2; ++k1) {
                    uint32_t ql[2][2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        ql[0][i] = ld_word_at(b0, c * 64 + k1 * 32 + 16 * i + 4 * t, sh0);
                        ql[1][i] = ld_word_at(b1, c * 64 + k1 * 32 + 16 * i + 4 * t, sh1);
                    }
#pragma unroll
                    for (int nib = 0; nib < 2; ++nib) {
                        const int k = k1 + 2 * nib;
                        uint32_t v[2][2];
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                v[r][i] = ((ql[r][i] >> (4 * nib)) & 0x0F0F0F0Fu) |
                                          ((k <= 2 ? q[r][i] << (4 - 2 * k) : q[r][i] >> 2) & 0x30303030u);
                        group(4 * c + k, v);
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int g = 4 * c + k;
                    uint32_t v[2][2];
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            v[r][i] = ((q[r][i] >> (2 * k)) & 0x03030303u) | ((g <= 2 ? hm[r][i] << (2 - g) : hm[r][i] >> (g - 2)) & 0x04040404u);
                    group(g, v);
                }
            }
        }
    }
};
template <int NT> struct SmallBlock<QT_Q6_K, NT> : SmallScaled16<QT_Q6_K, NT> {};
template <int NT> struct SmallBlock<QT_Q3_K, NT> : SmallScaled16<QT_Q3_K, NT> {};

// IQ2_S: thread t of a quad takes codebook group 4 g + t of 32-weight group g (8 weights, one sign
// byte); fragments are bf16(+-magnitude * 3 (2 scale + 1)), the block scale is d / 24.  The factor 3 costs
// nothing and rounds the magnitudes' products (8, 25, 43 times an odd number) least: weights are 1.44e-3 off
// in the 2-norm of a uniformly drawn payload, 1.69e-3 without it, 1.64e-3 in the GEMM, whose products have the
// block scale in them.  Exact products (a second bf16 part, or a mma per scale) cost 20 to 30 %.
template <int NT> struct SmallBlock<QT_IQ2_S, NT> {
    __device__ static __forceinline__ void run(uint32_t p0, uint32_t p1, uint32_t frag, uint32_t, uint32_t grid, int lane, float (&tot)[NT][4]) {
        const int t = lane & 3;
        const uint32_t p[2] = {p0, p1};
        uint32_t qh[2][2], sc[2][2];   // [row][groups 4 j .. 4 j + 3]
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            ld_words<2>(p[r] + 66, qh[r]);
            ld_words<2>(p[r] + 74, sc[r]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                qh[r][j] >>= 2 * t;                                                             // this thread's two index bits lowest
                sc[r][j] = ((sc[r][j] >> (4 * (t >> 1))) & 0x0F0F0F0Fu) * 6u + 0x03030303u;     // 3 (2 scale + 1)
            }
        }
        const float d0 = half_bits_to_float(lds16(p0)) * (1.0f / 24.0f), d1 = half_bits_to_float(lds16(p1)) * (1.0f / 24.0f);
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            uint32_t a[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t lo = lds8(p[r] + 2 + 4 * g + t);
                const uint32_t sg = lds8(p[r] + 34 + 4 * g + t) * 0x8001u;   // sign bit e at bits e and 15 + e
                const uint32_t idx = ((qh[r][g >> 2] >> (8 * (g & 3))) & 3u) << 8 | lo;
                const uint2 m = lds64(grid + idx * 8);
                const uint32_t s = hadd2_bf16(__byte_perm(sc[r][g >> 2], kTop128, 0x4040u + 0x0101u * (g & 3)), kMinus128);
                // weights 2 p, 2 p + 1: their sign bits moved onto the halves' sign bits
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t w = i == 0 ? m.x : m.y;
                    const uint32_t u = hadd2_bf16(bytes01(w, kTop128), kMinus128), v = hadd2_bf16(bytes23(w, kTop128), kMinus128);
                    a[i][r] = hmul2_bf16(u ^ ((sg << (15 - 4 * i)) & 0x80008000u), s);
                    a[i][2 + r] = hmul2_bf16(v ^ ((sg << (13 - 4 * i)) & 0x80008000u), s);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 x = lds128(frag + (g * NT + nt) * 512);
                mma_bf16(acc[nt], a[0], x.x, x.y);
                mma_bf16(acc[nt], a[1], x.z, x.w);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) add_scaled(tot[nt], d0, d1, acc[nt]);
    }
};

// Token tile `tile` of the call: expert, first row, tokens.
struct SmallTile {
    int expert, row0, ntok;
};

// Prefix sum over the groups (the CTA's whole work list): per group the cumulative number of tiles
// of `tok` tokens, first row and expert, in shared memory.  Invalid and empty groups have no tiles.
// Every thread returns the total.
__device__ __forceinline__ int small_scan_groups(const SmallArgs& a, int tok, int* cum, int* beg_s, int* exp_s, int* warp_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int base = 0;
    for (int g0 = 0; g0 < a.groups; g0 += blockDim.x) {
        const int g = g0 + threadIdx.x;
        int nt = 0, beg = 0;
        long long e = -1;
        if (g < a.groups) {
            e = a.experts[g];
            const int end = a.offsets[g];
            beg = g > 0 ? a.offsets[g - 1] : 0;
            if (e >= 0 && e < a.num_experts && beg >= 0 && beg < end && end <= a.rows) nt = (end - beg + tok - 1) / tok;
        }
        int incl = nt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += v;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        int before = base, all = base;
        for (int w = 0; w < nwarps; ++w) {
            const int s = warp_sum[w];
            if (w < warp) before += s;
            all += s;
        }
        if (g < a.groups) {
            cum[g] = before + incl;
            beg_s[g] = beg;
            exp_s[g] = static_cast<int>(e);
        }
        base = all;
        __syncthreads();
    }
    return base;
}

// `cum`: the three lists of small_scan_groups, one after the other
__device__ __forceinline__ SmallTile small_tile_at(const SmallArgs& a, int tok, const int* cum, int tile) {
    SmallTile r;
    if (a.experts == nullptr) {
        r.expert = 0;
        r.row0 = tile * tok;
        r.ntok = min(tok, a.rows - r.row0);
        return r;
    }
    int lo = 0, hi = a.groups - 1;   // first group whose cumulative count exceeds the tile
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] > tile) hi = mid; else lo = mid + 1;
    }
    const int first = lo > 0 ? cum[lo - 1] : 0;
    r.expert = cum[2 * a.groups + lo];
    r.row0 = cum[a.groups + lo] + (tile - first) * tok;
    r.ntok = min(tok, a.offsets[lo] - r.row0);
    return r;
}

// A CTA's range of the (token tile, weight set, group of rw row tiles) units; a unit's coordinates
// advance by carries, without divisions.
struct SmallWalk {
    struct Unit {
        int u, tile, set, rg;
    };
    int rtg, lo, hi;
    __device__ __forceinline__ SmallWalk(const SmallArgs& a, int ntiles) {
        rtg = (a.out_features + 16 * a.rw - 1) / (16 * a.rw);   // row-tile groups of a weight set
        // = units * b / ctas.  The host has checked that an int holds the units; a dense call's CTA often has one
        // unit, and two 64-bit divisions before its first load are 0.4 us of 8.7 (grouped: measured no gain)
        const int units = ntiles * rtg * a.nsets, ctas = gridDim.x, b = blockIdx.x;
        if (a.experts == nullptr) {
            const int each = units / ctas, more = units - each * ctas;
            lo = each * b + more * b / ctas;
            hi = each * (b + 1) + more * (b + 1) / ctas;
        } else {
            lo = static_cast<int>(static_cast<long long>(units) * b / ctas);
            hi = static_cast<int>(static_cast<long long>(units) * (b + 1) / ctas);
        }
    }
    __device__ __forceinline__ Unit first(const SmallArgs& a) const {
        Unit w;
        w.u = lo;
        w.tile = lo / (rtg * a.nsets);
        w.set = (lo - w.tile * rtg * a.nsets) / rtg;
        w.rg = lo - (w.tile * a.nsets + w.set) * rtg;
        return w;
    }
    __device__ __forceinline__ void advance(const SmallArgs& a, Unit& w) const {
        ++w.u;
        if (++w.rg == rtg) {
            w.rg = 0;
            if (++w.set == a.nsets) { w.set = 0; ++w.tile; }
        }
    }
};

// 16 weight rows x 8 tokens as the GEMM computes them: weights decoded to bf16, times x, summed in fp32.
//   off: byte of the first row in the tensor; last: its last row that exists (0..15); x: the first of ntok tokens
//   stage: a stage of this warp, none in flight; v: the elements of this thread's mma fragment
template <int QT>
__device__ __forceinline__ void small_direct(const uint8_t* wgt, long long wgt_bytes, long long off, int row_bytes, int last, int nkb,
                                          const __nv_bfloat16* x, int ntok, uint32_t stage, uint32_t grid, float (&v)[4]) {
    using Fmt = BlockFmt<QT>;
    using Sf = SmallFmt<QT>;
    const int lane = threadIdx.x & 31, row = lane & 15, half = lane >> 4, K = nkb * 256;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int kb = 0; kb < nkb; ++kb) {
        __syncwarp();
        for (int c = lane; c < 16 * Sf::kChunks; c += 32) {
            const int r = c / Sf::kChunks, po = (c - r * Sf::kChunks) * 16;
            const long long at = ((off + static_cast<long long>(min(r, last)) * row_bytes + kb * Fmt::kBytes) & ~15LL) + po;
            const int n = static_cast<int>(max(0LL, min(16LL, wgt_bytes - at)));
            cp_async16(stage + r * Sf::kPitch + po, n > 0 ? wgt + at : wgt, n);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        const long long at = off + static_cast<long long>(min(row, last)) * row_bytes + kb * Fmt::kBytes;
        const uint32_t blk = stage + row * Sf::kPitch + static_cast<uint32_t>(at & 15);
#pragma unroll 1
        for (int g = 4 * half; g < 4 * half + 4; ++g) {
            uint4 w[4];
            decode32<QT>(blk, g, grid, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= ntok) break;
                const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<long long>(j) * K + kb * 256 + g * 32);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 xs = src[c];
                    const uint32_t a[4] = {w[c].x, w[c].y, w[c].z, w[c].w}, b[4] = {xs.x, xs.y, xs.z, xs.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 wf = __bfloat1622float2(as_bf162(a[i])), xf = __bfloat1622float2(as_bf162(b[i]));
                        acc[j] = fmaf(wf.x, xf.x, acc[j]);
                        acc[j] = fmaf(wf.y, xf.y, acc[j]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float sum = acc[j] + __shfl_xor_sync(0xFFFFFFFFu, acc[j], 16);
        const float lo = __shfl_sync(0xFFFFFFFFu, sum, lane >> 2), hi = __shfl_sync(0xFFFFFFFFu, sum, (lane >> 2) + 8);
        if ((j >> 1) == (lane & 3)) { v[j & 1] = lo; v[2 + (j & 1)] = hi; }
    }
}
__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7F800000u) == 0x7F800000u; }

// After the kernel's walk: every thread looks again at the results that it stored and replaces those
// that are not finite.
template <int QT, int NT>
__device__ __forceinline__ void small_redo(const SmallArgs& args, int ntiles, const int* cum, uint32_t my_ring, uint32_t grid_s) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int kw = args.kw, rw = args.rw, rwi = warp / kw, ks = warp - rwi * kw;
    const int N = args.out_features, K = args.in_features;
    const SmallWalk walk(args, ntiles);
    int turn = 0;   // as in the kernel: the thread that stored a result reads it back
    for (SmallWalk::Unit un = walk.first(args); un.u < walk.hi; walk.advance(args, un)) {
        const SmallTile ct = small_tile_at(args, 8 * NT, cum, un.tile);
        const int row0 = (un.rg * rw + rwi) * 16;
        for (int nt = 0; nt < NT; ++nt) {
            const bool mine = ks == turn;
            if (++turn == kw) turn = 0;
            if (!mine || nt * 8 >= ct.ntok || row0 >= N) continue;
            __nv_bfloat16* at[4];
            bool redo[4], any = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int token = nt * 8 + 2 * t + (j & 1), row = row0 + g + 8 * (j >> 1), r = ct.row0 + token;
                at[j] = nullptr;
                if (token < ct.ntok && row < N) {
                    at[j] = args.out_rows != nullptr ? args.out_rows[r] : args.out[un.set] + static_cast<long long>(r) * N;
                    if (at[j] != nullptr) at[j] += row;
                }
                redo[j] = at[j] != nullptr && not_finite(__bfloat162float(*at[j]));
                any |= redo[j];
            }
            if (!__any_sync(0xFFFFFFFFu, any)) continue;
            float v[4];
            small_direct<QT>(args.wgt[un.set], args.wgt_bytes, (static_cast<long long>(ct.expert) * N + row0) * args.row_bytes, args.row_bytes,
                             min(15, N - 1 - row0), K >> 8, args.act + static_cast<long long>(ct.row0 + nt * 8) * K, ct.ntok - nt * 8, my_ring,
                             grid_s, v);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (redo[j]) *at[j] = __float2bfloat16(v[j]);
        }
    }
}

// the same as a call, for the kernels that have no register to spare (us inlined / called: 600 tokens, Q3_K
// experts, 24 tokens per tile 311.6 / 308.8; 16 tokens, IQ2_S experts, 8 per tile 101.7 / 103.7)
template <int QT, int NT>
__device__ __noinline__ void small_redo_call(const SmallArgs& args, int ntiles, const int* cum, uint32_t my_ring, uint32_t grid_s) {
    small_redo<QT, NT>(args, ntiles, cum, my_ring, grid_s);
}

template <int QT, int NT>
__global__ void __launch_bounds__(kSmallWarps * 32, 1) mmq_small_kernel(const __grid_constant__ SmallArgs args) {
    using Fmt = BlockFmt<QT>;
    using Sf = SmallFmt<QT>;
    constexpr int kTok = 8 * NT;
    constexpr int kPer = (16 * Sf::kChunks + 31) / 32;   // 16-byte pieces of a stage per lane
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int kw = args.kw, rw = args.rw, S = args.stages;
    const int rwi = warp / kw, ks = warp - rwi * kw;
    const int N = args.out_features, K = args.in_features, nkb = K >> 8, row_bytes = args.row_bytes;
    const int g = lane >> 2, t = lane & 3;

    const uint32_t frag_s = smem_u32(smem);
    const uint32_t sums_s = frag_s + nkb * NT * 4096;
    const uint32_t grid_s = sums_s + nkb * NT * Sf::kSumBytes;
    const uint32_t ring_s = grid_s + Sf::kGridBytes;
    const uint32_t red_s = ring_s + nwarps * S * Sf::kStageBytes;
    int* const lists = reinterpret_cast<int*>(smem + (red_s - frag_s) + (kw > 1 ? 2 * nwarps * NT * 512 : 0));
    int* const warp_sum = lists;                     // kSmallWarps
    int* const cum = lists + kSmallWarps;            // per group: tiles up to its end, first row, expert

    int ntiles;
    if (args.experts != nullptr) ntiles = small_scan_groups(args, kTok, cum, cum + args.groups, cum + 2 * args.groups, warp_sum);
    else ntiles = (args.rows + kTok - 1) / kTok;
    if (args.tile_count != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *args.tile_count = ntiles;
    auto tile_of = [&](int tile) { return small_tile_at(args, kTok, cum, tile); };

    const SmallWalk walk(args, ntiles);
    const int hi = walk.hi;
    using Unit = SmallWalk::Unit;
    const Unit first = walk.first(args);
    auto advance = [&](Unit& w) { walk.advance(args, w); };

    if (Sf::kGridBytes) {
        for (int i = threadIdx.x; i < 1024; i += blockDim.x) reinterpret_cast<uint64_t*>(smem + (grid_s - frag_s))[i] = args.iq2s_grid[i];
    }

    // ---- loads: a walk over (unit, block) of this warp, ahead of the one that computes.  The lanes
    // copy the 16-byte pieces of the 16 windows in order, so that a request covers few lines.
    const uint32_t my_ring = ring_s + warp * S * Sf::kStageBytes;
    int src_of[kPer];        // piece i of this lane: offset from the window of the tile's first row
    uint32_t dst_of[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int c = lane + 32 * i, r = c / Sf::kChunks, o = (c - r * Sf::kChunks) * 16;
        src_of[i] = r * row_bytes + o;
        dst_of[i] = my_ring + r * Sf::kPitch + o;
    }
    const bool rows_aligned = Fmt::kAligned || (row_bytes & 15) == 0;   // all rows of a tile are misaligned alike
    Unit pu = first;
    int pkb = ks, p_expert = -1, p_tile = -1;
    bool p_new = true, p_plain = false;
    const uint8_t* p_base = nullptr;   // 16-byte aligned address at or below the unit's first row
    int p_off = 0;                     // its current block from there
    long long p_left = 0;              // bytes from p_base to the end of the tensor
    uint32_t p_slot = 0;
    auto issue = [&]() {
        if (pu.u < hi) {
            if (p_new) {
                if (pu.tile != p_tile) { p_expert = tile_of(pu.tile).expert; p_tile = pu.tile; }
                const int row = min((pu.rg * rw + rwi) * 16, N - 1);
                const long long off = (static_cast<long long>(p_expert) * N + row) * row_bytes;
                p_base = args.wgt[pu.set] + (off & ~15LL);
                p_left = args.wgt_bytes - (off & ~15LL);
                p_off = static_cast<int>(off & 15) + ks * Fmt::kBytes;
                // whole tile, not the tensor's last rows: every piece is at its usual place and readable
                p_plain = rows_aligned && row + 16 <= N && (Fmt::kAligned || p_left >= 17LL * row_bytes);
                p_new = false;
            }
            const uint32_t ring_off = p_slot * Sf::kStageBytes;
            if (p_plain) {
                const uint8_t* src = p_base + (p_off & ~15);
#pragma unroll
                for (int i = 0; i < kPer; ++i)
                    if (lane + 32 * i < 16 * Sf::kChunks) cp_async16(dst_of[i] + ring_off, src + src_of[i], 16);
            } else {
                const int last = N - 1 - min((pu.rg * rw + rwi) * 16, N - 1);
                for (int c = lane; c < 16 * Sf::kChunks; c += 32) {
                    const int r = c / Sf::kChunks, po = (c - r * Sf::kChunks) * 16;
                    const int o = ((p_off + min(r, last) * row_bytes) & ~15) + po;
                    const int n = static_cast<int>(max(0LL, min(16LL, p_left - o)));   // nothing is read past the tensor
                    cp_async16(my_ring + r * Sf::kPitch + po + ring_off, n > 0 ? p_base + o : p_base, n);
                }
            }
            if (++p_slot == static_cast<uint32_t>(S)) p_slot = 0;
            pkb += kw;
            p_off += kw * Fmt::kBytes;
            if (pkb >= nkb) { pkb = ks; advance(pu); p_new = true; }
        }
        cp_async_commit();
    };
    for (int s = 0; s < S - 1; ++s) issue();

    uint32_t slot = 0, parity = 0;
    int cur_tile = -1, turn = 0;
    SmallTile ct = {0, 0, 0};
    // stays zero while this thread's results are finite: infinities and NaN times zero are NaN.  (Two
    // instructions per 8 tokens; tests of each result cost 1-4 % where the reduction has two blocks.)
    float2 odd = make_float2(0.f, 0.f);
    for (Unit un = first; un.u < hi; advance(un)) {
        if (un.tile != cur_tile) {
            // ---- x of the token tile as mma fragments
            if (cur_tile >= 0) __syncthreads();
            cur_tile = un.tile;
            ct = tile_of(un.tile);
            const __nv_bfloat16* x = args.act + static_cast<long long>(ct.row0) * K;
#pragma unroll 4
            for (int q = warp; q < nkb * 8 * NT; q += nwarps) {
                const int g32 = q / NT, nt = q - g32 * NT, token = nt * 8 + g;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (token < ct.ntok) {
                    const __nv_bfloat16* src = x + static_cast<long long>(token) * K + g32 * 32;
                    if (Sf::kPairOrder) {
                        v = *reinterpret_cast<const uint4*>(src + 8 * t);
                    } else {
                        const uint2 a = *reinterpret_cast<const uint2*>(src + 4 * t), b = *reinterpret_cast<const uint2*>(src + 16 + 4 * t);
                        v = make_uint4(a.x, a.y, b.x, b.y);
                    }
                }
                sts128(frag_s + q * 512 + lane * 16, v);
                if (Sf::kSumBytes) {   // sums of the tokens over each scale group, as the B operand of the offsets' mma
                    const float2 f0 = __bfloat1622float2(as_bf162(v.x)), f1 = __bfloat1622float2(as_bf162(v.y));
                    const float2 f2 = __bfloat1622float2(as_bf162(v.z)), f3 = __bfloat1622float2(as_bf162(v.w));
                    float s0 = (f0.x + f0.y) + (f1.x + f1.y), s1 = (f2.x + f2.y) + (f3.x + f3.y);
                    if (Sf::kAffine) s0 += s1;
                    s0 += __shfl_xor_sync(0xFFFFFFFFu, s0, 1);
                    s0 += __shfl_xor_sync(0xFFFFFFFFu, s0, 2);
                    if (!Sf::kAffine) {
                        s1 += __shfl_xor_sync(0xFFFFFFFFu, s1, 1);
                        s1 += __shfl_xor_sync(0xFFFFFFFFu, s1, 2);
                    }
                    if (t < (Sf::kAffine ? 1 : 2)) {   // lane t writes the sum of group (affine) or half-group t
                        const float s = t == 0 ? s0 : s1;
                        const int at = Sf::kAffine ? g32 & 7 : 2 * (g32 & 7) + t;   // scale group inside the block
                        const __nv_bfloat16 s_hi = __float2bfloat16(s), s_lo = __float2bfloat16(s - __bfloat162float(s_hi));
                        __nv_bfloat16* m = reinterpret_cast<__nv_bfloat16*>(smem + (sums_s - frag_s) + ((g32 >> 3) * NT + nt) * Sf::kSumBytes +
                                                                            (g * 4 + (at >> 2)) * 8 + (at & 3) * 2);
                        m[0] = s_hi;
                        m[Sf::kAffine ? 8 : 128] = s_lo;   // two lanes further on, or in the second mma's fragment
                    }
                }
            }
            __syncthreads();
        }
        float tot[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) tot[nt][0] = tot[nt][1] = tot[nt][2] = tot[nt][3] = 0.f;
        const int row0 = (un.rg * rw + rwi) * 16;
        uint32_t at0 = 0, at1 = 0;   // misalignment of this thread's two rows, before the block's offset
        if (!Fmt::kAligned) {
            const int row = min(row0, N - 1), last = N - 1 - row;
            const uint32_t first_at = (static_cast<uint32_t>(ct.expert) * N + row) * row_bytes;   // only the low bits matter
            at0 = first_at + min(g, last) * row_bytes;
            at1 = first_at + min(g + 8, last) * row_bytes;
        }
        for (int kb = ks; kb < nkb; kb += kw) {
            if (S == 4) cp_async_wait<2>(); else if (S == 3) cp_async_wait<1>(); else cp_async_wait<0>();
            __syncwarp();
            issue();
            uint32_t p0 = my_ring + slot * Sf::kStageBytes + g * Sf::kPitch, p1 = p0 + 8 * Sf::kPitch;
            if (++slot == static_cast<uint32_t>(S)) slot = 0;
            if (!Fmt::kAligned) {
                p0 += (at0 + kb * Fmt::kBytes) & 15;
                p1 += (at1 + kb * Fmt::kBytes) & 15;
            }
            SmallBlock<QT, NT>::run(p0, p1, frag_s + kb * NT * 4096 + lane * 16, sums_s + kb * NT * Sf::kSumBytes + lane * 8, grid_s, lane, tot);
        }
        // ---- the slices' partial sums meet; the next unit uses the other buffer.  The warps of a row
        // tile take turns (per 8 tokens) at adding and storing.
        const uint32_t red = red_s + (parity * nwarps + rwi * kw) * NT * 512;
        parity ^= 1u;
        if (kw > 1) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
                sts128(red + (ks * NT + nt) * 512 + lane * 16, make_uint4(__float_as_uint(tot[nt][0]), __float_as_uint(tot[nt][1]),
                                                                         __float_as_uint(tot[nt][2]), __float_as_uint(tot[nt][3])));
            bar_named(rwi + 1, kw * 32);   // kw > 1: at most 8 row tiles
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const bool mine = ks == turn;
            if (++turn == kw) turn = 0;
            if (!mine) continue;
            float v[4] = {tot[nt][0], tot[nt][1], tot[nt][2], tot[nt][3]};
            if (kw > 1) {
                v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll 4
                for (int i = 0; i < kw; ++i) {
                    const uint4 p = lds128(red + (i * NT + nt) * 512 + lane * 16);
                    v[0] += __uint_as_float(p.x);
                    v[1] += __uint_as_float(p.y);
                    v[2] += __uint_as_float(p.z);
                    v[3] += __uint_as_float(p.w);
                }
            }
            odd = __ffma2_rn(make_float2(v[0], v[1]), make_float2(0.f, 0.f), odd);
            odd = __ffma2_rn(make_float2(v[2], v[3]), make_float2(0.f, 0.f), odd);
            const int token = nt * 8 + 2 * t;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (token + j < ct.ntok) {
                    const int r = ct.row0 + token + j;
                    __nv_bfloat16* dst = args.out_rows != nullptr ? args.out_rows[r] : args.out[un.set] + static_cast<long long>(r) * N;
                    if (dst != nullptr && row0 + g < N) dst[row0 + g] = __float2bfloat16(v[j]);
                    if (dst != nullptr && row0 + g + 8 < N) dst[row0 + g + 8] = __float2bfloat16(v[2 + j]);
                }
            }
        }
    }
    cp_async_wait<0>();
    if (__any_sync(0xFFFFFFFFu, odd.x != 0.f || odd.y != 0.f)) {
        if constexpr (NT <= 2) small_redo<QT, NT>(args, ntiles, cum, my_ring, grid_s);
        else small_redo_call<QT, NT>(args, ntiles, cum, my_ring, grid_s);
    }
}

}  // namespace tgo
