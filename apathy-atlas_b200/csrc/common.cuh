// Shared device helpers: BF16 packing, the NVFP4 codecs, the device status word.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace atlas {

// ---- device status word -------------------------------------------------------------------
// First problem recorded by any kernel since the last clear (0 = clean).  Kernels never trap:
// they record a code here and carry on in a defined way (treat the row as un-adapted, or
// leave the tile unwritten after a wait that expired).
enum : uint32_t {
    STATUS_OK = 0,
    STATUS_SLOT_OUT_OF_RANGE = 1,   // seq_slot[i] >= max_loras
    STATUS_NEGATIVE_SCALE = 2,      // FP4-activation mode met a weight scale byte with its sign bit set; the sign was dropped
    STATUS_TILE_CAPACITY = 3,       // the shrink met more (slot, granule) pairs in a token tile than its tile output reserves
    STATUS_WAIT_EXPIRED_PRODUCER = 0x100,
    STATUS_WAIT_EXPIRED_DEQUANT = 0x101,
    STATUS_WAIT_EXPIRED_MMA = 0x102,
    STATUS_WAIT_EXPIRED_EPILOGUE = 0x103,
};

__device__ uint32_t g_status_word = 0;

__device__ __forceinline__ void record_status(uint32_t code) { atomicCAS(&g_status_word, 0u, code); }

// ---- programmatic dependent launch ------------------------------------------------------------
// A decode step is a chain of short kernels, and between two of them an ordinary launch leaves the machine idle for a few
// microseconds.  A kernel may (a) release the next launch once all its own CTAs run, and (b) be launched as a dependent, which may
// then start early and has to wait until everything before it in the stream has completed and is visible.
//   launched as dependents     both tensor-core shrinks, the main kernel behind a shrink and without adapters, the tensor-core expand, the
//                              dense linear, the QKV consumers, SwiGLU in both forms, the quantiser
//   releasing                  all of these but lora_shrink_mma_kernel and lora_shrink_grouped_kernel, which do so only in front of a
//                              main kernel or of the dense linear
//   neither                    a main kernel over a t that an earlier call left, and the small-batch kernel for more than eight tokens without
//                              adapters, release but are launched in order; the NVFP4 decode, the maximum, the CUDA-core linear and
//                              expand do neither
// A dependent begins with the wait, with three exceptions:
//   the main kernel and the dense linear behind their shrink read x, weights and routing ahead of it: that shrink has waited before
//   releasing them; they wait before they read t, or before they end, on every path, so that nothing behind them overtakes the shrink;
//   the main kernel without adapters, its scales by TMA or from rows: only the warps that read memory begin with the wait, and the others
//   work on what those bring;
//   lora_shrink_mma_kernel looks at seq_slot, a_table and rank_table while the kernel ahead may still be writing them.  Those values
//   only choose lines of A to prefetch, out of the declared pool alone; they are read past the first-level cache, and everything is
//   read again behind the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The pointer as a value that does not exist before this point: keeps read-only loads through it behind pdl_wait().
template <typename T> __device__ __forceinline__ T* pdl_after(T* p) {
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}

// ---- BF16 <-> FP32 ---------------------------------------------------------------------------
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ uint16_t f32_to_bf16_bits(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);               // one conversion for the pair, each rounded to nearest even
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- E2M1 / E4M3, scalar forms (bit-for-bit the arithmetic of
//      kernels/gb10/common/dequant_nvfp4_bf16.cu:26-46) ---------------------------------------
__device__ __forceinline__ float e2m1_decode(uint32_t nib) {
    // magnitude = {0, .5, 1, 1.5, 2, 3, 4, 6}[nib & 7], bit 3 = sign
    const uint32_t m = nib & 7u;
    // FP32 bits with (m << 22) are 2^(e-127)*(1+mant/2) for e>0 and a subnormal for e==0;
    // multiplying by 2^126 gives the E2M1 value exactly in both cases.
    float v = __uint_as_float(m << 22) * 8.507059173023462e37f;   // 2^126
    return (nib & 8u) ? -v : v;
}

__device__ __forceinline__ float e4m3_decode(uint32_t b) {
    const uint32_t e = (b >> 3) & 0xFu, m = b & 0x7u;
    float v;
    if (e == 0u) v = float(m) * 0.001953125f;
    else if (e == 15u && m == 7u) v = 0.0f;               // the NaN byte decodes to 0
    else v = __uint_as_float(((e + 120u) << 23) | (m << 20));
    return (b & 0x80u) ? -v : v;
}

// ---- packed BF16x2 multiply (subnormal inputs are honoured: no .ftz) ------------------------
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// The expansion is bound by the integer pipe (shifts, logic and permutes issue at half rate), so positions are reached by
// multiplications, which the FMA pipe does beside it: a nibble n in each half of a word, times 0x1040, has its sign at bit 15
// (n << 12) and its three magnitude bits at bits 6 to 8 (n << 6), the BF16 exponent's last two and the mantissa's first:
// value * 2^-126, subnormal included.
constexpr uint32_t kE2m1At = 0x1040u, kE2m1Bits = 0x81C081C0u;

// Four E4M3 scale bytes with NaN bytes (0x7F, 0xFF) replaced by zeros of their sign.
__device__ __forceinline__ uint32_t e4m3x4_clear_nan(uint32_t w) {
    const uint32_t nan = (((w & 0x7F7F7F7Fu) + 0x01010101u) & 0x80808080u) >> 7;
    return w ^ (nan * 0x7Fu);
}
// Bytes i0 and i1 of `w` (no NaN), chosen by sel = i0 | 4 << 4 | i1 << 8 | 4 << 12, as BF16x2 multipliers {f, f} with f = e4m3 * 2^118.
// (byte & 0x7F) << 4 read as BF16 is e4m3 * 2^-120 for normals and subnormals alike.
__device__ __forceinline__ void e4m3x2_to_bf16x2_shifted(uint32_t w, uint32_t sel, uint32_t& f0, uint32_t& f1) {
    const uint32_t b = prmt(w, 0u, sel);
    uint32_t v = ((b * 0x10u) & 0x07F007F0u) | ((b * 0x100u) & 0x80008000u);
    v = bf16x2_mul(v, 0x7B807B80u);   // * 2^120 : exact E4M3 value
    v = bf16x2_mul(v, 0x7A807A80u);   // * 2^118
    f0 = prmt(v, 0u, 0x1010u);
    f1 = prmt(v, 0u, 0x3232u);
}

// Eight E2M1 codes (element i in bits [4i, 4i+4)) times a BF16x2 multiplier {f, f}
// -> eight BF16 values in element order, as four BF16x2 words.
// With f = scale * 2^118 each output is E2M1 * scale * 2^-8, exact in BF16 (<= 6 significant bits).
__device__ __forceinline__ void e2m1x8_to_bf16x8(uint32_t p, uint32_t mul, uint32_t (&out)[4]) {
    const uint32_t even = p & 0x0F0F0F0Fu, odd = (p >> 4) & 0x0F0F0F0Fu;
    // byte i of both, one to each half of a word; the bytes between are the (clear) sign bits of the same bytes
    out[0] = bf16x2_mul((prmt(even, odd, 0xC480u) * kE2m1At) & kE2m1Bits, mul);
    out[1] = bf16x2_mul((prmt(even, odd, 0xD591u) * kE2m1At) & kE2m1Bits, mul);
    out[2] = bf16x2_mul((prmt(even, odd, 0xE6A2u) * kE2m1At) & kE2m1Bits, mul);
    out[3] = bf16x2_mul((prmt(even, odd, 0xF7B3u) * kE2m1At) & kE2m1Bits, mul);
}
// The same without the order: words of the pairs (i, i + 4), which need no permutes.
__device__ __forceinline__ void e2m1x8_to_pairs(uint32_t p, uint32_t mul, uint32_t (&h)[4]) {
    const uint32_t q = p >> 8;
    h[0] = bf16x2_mul(((p & 0x000F000Fu) * kE2m1At) & kE2m1Bits, mul);
    h[1] = bf16x2_mul(((p & 0x00F000F0u) * (kE2m1At >> 4)) & kE2m1Bits, mul);
    h[2] = bf16x2_mul(((q & 0x000F000Fu) * kE2m1At) & kE2m1Bits, mul);
    h[3] = bf16x2_mul(((q & 0x00F000F0u) * (kE2m1At >> 4)) & kE2m1Bits, mul);
}

constexpr float kWeightPreScale = 256.0f;   // 2^8: weights enter the MMA as value * 2^-8

}  // namespace atlas
