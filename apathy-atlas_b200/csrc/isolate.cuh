// Keeps adapters apart in the fused kernels, for the shapes whose LoRA term was once added row by row (K not a multiple of 256,
// ranks above 64: Params::isolate).
//
// A fused kernel multiplies every B_s that occurs in a token tile with all of the tile's tokens, zeros standing for t of those
// routed elsewhere.  Zero times an infinity or a NaN is a NaN: one adapter with a non-finite element in row f of its B makes a
// NaN of feature f for the whole tile.  That NaN survives every later addition, so it is enough to look for NaNs in what is
// stored: a CTA that has stored one computes again, behind its last store, what a row's own x, A and B leave finite.
//
// The look costs three integer operations per two outputs and one barrier (77 tokens x 2880 features x 2880: 17.2 us with it,
// 17.0 without; as a kernel of its own behind the main one 19.3).  It is compiled into instances of their own (ISO): in all of them
// it cost the calls of other shapes 0.5 to 1.3 %.  A NaN costs a dot product of length K per output concerned, by one warp.
#pragma once

#include "common.cuh"

namespace atlas {

// bits 15 and 31 are set where the two BF16 values of w are NaNs (the sum of several such words may be ORed before masking)
__device__ __forceinline__ uint32_t bf16x2_nan_bits(uint32_t w) { return (w & 0x7FFF7FFFu) + 0x007F007Fu; }
constexpr uint32_t kNanBits = 0x80008000u;
__device__ __forceinline__ bool bf16_nan(uint32_t bits) { return (bits & 0x7FFFu) > 0x7F80u; }
__device__ __forceinline__ bool bf16_not_finite(uint32_t bits) { return (bits & 0x7F80u) == 0x7F80u; }
__device__ __forceinline__ float bf16_value(uint32_t bits) { return __uint_as_float(bits << 16); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Row m of [f_lo, f_hi) holds a NaN.  `t_s`: shared memory for max_rank BF16 values.  By all threads of the CTA.
template <typename P>
__device__ __forceinline__ void isolate_row(const P& p, uint32_t m, uint32_t f_lo, uint32_t f_hi, uint16_t* t_s) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x, warps = threads >> 5;
    const uint16_t* x = p.x + size_t(m) * p.x_row_stride;
    bool own = false;
    for (uint32_t k = tid; k < p.K; k += threads) own |= bf16_not_finite(x[k]);
    if (__syncthreads_or(own)) return;                                   // the token's own

    const int32_t s = p.seq_slot[m];
    const uint16_t* B = nullptr;
    uint32_t rank = 0;
    if (s >= 0 && uint32_t(s) < p.max_loras && p.a_table[s] != 0ull && p.b_table[s] != 0ull) {
        const uint16_t* A = reinterpret_cast<const uint16_t*>(p.a_table[s]);
        B = reinterpret_cast<const uint16_t*>(p.b_table[s]);
        rank = p.rank_table ? min(p.rank_table[s], p.max_rank) : p.max_rank;
        const float f = p.scale_table[s] * p.post;
        for (uint32_t j = warp; j < rank; j += warps) {
            float sum = 0.0f;
            for (uint32_t k = lane; k < p.K; k += 32) sum = fmaf(bf16_value(x[k]), bf16_value(A[size_t(j) * p.K + k]), sum);
            sum = warp_sum(sum);
            if (lane == 0) t_s[j] = f32_to_bf16_bits(sum * f);
        }
    }
    __syncthreads();
    own = false;
    for (uint32_t j = tid; j < rank; j += threads) own |= bf16_not_finite(t_s[j]);
    if (__syncthreads_or(own)) return;                                   // its adapter's, through A

    uint16_t* y = p.y + size_t(m) * p.out_row_stride;
    for (uint32_t f = f_lo + warp; f < f_hi; f += warps) {
        if (!bf16_nan(__ldcg(y + f))) continue;
        float sum = 0.0f;
        own = false;
        for (uint32_t j = lane; j < rank; j += 32) {
            const uint32_t b = B[size_t(f) * p.max_rank + j];
            own |= bf16_not_finite(b);
            sum = fmaf(bf16_value(t_s[j]), bf16_value(b), sum);
        }
        if (__any_sync(0xFFFFFFFFu, own)) continue;                      // its adapter's, through B
        const uint32_t* code = reinterpret_cast<const uint32_t*>(p.w_packed + size_t(f) * (p.K / 2));
        const uint8_t* scale = p.w_scale + size_t(f) * (p.K / 16);
        for (uint32_t i = lane; i < p.K / 8; i += 32) {
            const uint32_t w = code[i];
            const float sc = e4m3_decode(scale[i / 2]) * (1.0f / kWeightPreScale);
            const uint4 xv = *reinterpret_cast<const uint4*>(x + 8 * i);
            const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sum = fmaf(e2m1_decode((w >> (8 * e)) & 0xFu) * sc, bf16_lo(xw[e]), sum);
                sum = fmaf(e2m1_decode((w >> (8 * e + 4)) & 0xFu) * sc, bf16_hi(xw[e]), sum);
            }
        }
        sum = warp_sum(sum);
        if (lane == 0) y[f] = f32_to_bf16_bits(sum * p.out_scale);
    }
}

// (Inlined: as a call it made the kernels that use it spill in their K loops, up to 3 % of a call.)
// The tile [m_lo, m_hi) x [f_lo, f_hi) that this CTA has stored; of its 16-token chunks only every ks-th, from kz (split K).
template <typename P>
__device__ __forceinline__ void isolate_tile(const P& p, uint32_t m_lo, uint32_t m_hi, uint32_t f_lo, uint32_t f_hi, uint32_t ks, uint32_t kz,
                                          uint16_t* t_s) {
    for (uint32_t m = m_lo; m < m_hi; ++m) {
        if (((m - m_lo) / 16u) % ks != kz) continue;
        bool any = false;
        for (uint32_t f = f_lo + threadIdx.x; f < f_hi; f += blockDim.x) any |= bf16_nan(__ldcg(p.y + size_t(m) * p.out_row_stride + f));
        if (__syncthreads_or(any)) isolate_row(p, m, f_lo, f_hi, t_s);
        __syncthreads();                                                 // t_s is written again for the next row
    }
}

}  // namespace atlas
