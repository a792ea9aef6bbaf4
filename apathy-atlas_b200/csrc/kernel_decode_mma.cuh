// The fused NVFP4 + multi-LoRA linear for the smallest batches: weights expanded in registers, mma.sync.
//
//   y[m, f] = bf16( out_scale * ( sum_k W'[f,k] x[m,k] + sum_j B_s[f,j] t[m,j] ) ),   s = seq_slot[m], t pre-scaled by the shrink
//
// A decode batch is bound by streaming the weights once.  The tcgen05 form cannot keep up with that stream: its weight operand
// goes through tensor memory, which fixes the order of the K elements (four byte permutes per eight codes), and its
// eight expansion warps are busy for 344 cycles per 128 x 64 block whatever the batch: one token x 14336 features x 4096
// takes 17.7 us for 33 MB, 14.8 here.  Here every warp of the SM expands, the operand stays in the registers the
// codes were expanded in, and since BOTH operands of mma.sync come from registers the K elements may take any order as long as
// they meet their partners: the pairs (i, i + 4) that fall out of a word of eight codes are used as they are, and x is paired
// the same way (four permutes per eight elements of x, shared by all features of the warp).
//
// A CTA owns 16 * TILES features and all of K.  Interleaved 128-wide K steps make eight partial sums, one to each of eight warps or
// two to each of four (with as many more CTAs on an SM): the same bits, so that either form may be taken for any batch and pool, and
// a row without an adapter is the base call's.  Per thread and feature row a step is one 128-bit load of 32 codes and their two scale
// bytes, from global memory with the next step's loads in flight while one is multiplied, or (TMA) from a ring in shared memory that
// a warp of its own fills; the partial sums are added in their order through shared memory.  No cluster, no tensor memory; but for the
// ring's barriers, two.
// The MMA's M is 16 features, its N 8 tokens (NT of them side by side).
//
// LoRA: granule j (16 ranks) of slot s is one more K step of partial sum (s + 3 j) % 8, so that the order in which a token's terms
// are added depends on its own slot alone.  t rows come from the shrink this kernel may overtake (programmatic dependent
// launch): they are first read behind griddepcontrol.wait, after the base loop.
#pragma once

#include "kernel_shrink_mma.cuh"
#include "kernel_tc.cuh"

namespace atlas {

constexpr int DCM_SUMS = 8;          // partial sums of an output, whatever the number of warps
constexpr int DCM_KSTEP = 128;
constexpr int DCM_MAX_TOKENS = 16;

struct DecodeParams {
    const uint16_t* x;
    const uint8_t* w_packed;
    const uint8_t* w_scale;
    uint32_t x_row_stride;
};

// TMA form: the ring of a CTA, filled by a warp of its own.  A stage is a step of every warp: [16 TILES rows x 128 B] of codes for every two
// of them, swizzled, then their scale bytes [16 TILES rows x 8 WARPS B], swizzled over their own width.
template <int TILES, int WARPS> struct DcmRing {
    static constexpr int ROWS = 16 * TILES, BOXES = WARPS / 2;
    static constexpr int CODES = BOXES * ROWS * 128, SCALES = ROWS * 8 * WARPS;
    static constexpr int STAGE = (CODES + SCALES + 1023) / 1024 * 1024, STAGES = 4;
    static constexpr int SMEM_BYTES = STAGES * STAGE + 1024;
};

// TMA: codes and scales come through shared memory (decode_by_tma); the same bits.  BASE: no adapters, launched as a dependent of whatever
// is before it (instances of their own: the wait in all of them cost calls with adapters 1 to 2 %).  Those release late: a next grid
// that comes while this one's CTAs are all at work takes the places they happen to leave, and its SMs get unequal numbers of CTAs.  One
// token behind one another, launched in order / released at the start / behind the loop (us): 11008 x 4096 12.8 / 14.4 / 11.9, 2048 x
// 2048 2.8 / - / 2.4.  (Two n-tiles have no such instance: 12 tokens x 1280 x 17408 14.1 / 20.4 / 15.2.)  SELFTEST: nothing fills the ring, and every wait on it runs out.
template <int TILES, int NT, int WARPS, bool TMA, bool BASE, bool SELFTEST = false>
__global__ void __launch_bounds__(32 * (WARPS + (TMA ? 1 : 0)), 16 / WARPS)
nvfp4_lora_decode_mma_kernel(const DecodeParams w, const tc::Params p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s) {
    using R = DcmRing<TILES, WARPS>;
    constexpr int SETS = DCM_SUMS / WARPS;                             // partial sums of a warp
    static_assert(SETS * WARPS == DCM_SUMS && SETS <= 2, "two steps to a turn of the base loop, one for either sum");
    __shared__ float part[DCM_SUMS][NT * 8][TILES * 16 + 1];           // [partial sum][token][feature]
    __shared__ int32_t slot_s[DCM_MAX_TOKENS];
    __shared__ uint32_t rank_s[DCM_MAX_TOKENS];                        // of the slot in slot_s: its rank
    __shared__ uint64_t b_s[DCM_MAX_TOKENS];                           // and its B (read once, not granule by granule behind the shrink)
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t f0 = blockIdx.x * (TILES * 16);
    extern __shared__ uint8_t dcm_dyn[];
    __shared__ uint64_t bars[TMA ? 2 * R::STAGES : 1];
    __shared__ uint32_t abort_s;
    const uint32_t ring = (tc::smem_u32(dcm_dyn) + 1023u) & ~1023u, BAR_FULL = tc::smem_u32(bars), BAR_EMPTY = BAR_FULL + 8 * R::STAGES;
    volatile uint32_t* abort_flag = &abort_s;
    if constexpr (TMA) {
        if (tid == 0) {
            for (int i = 0; i < R::STAGES; ++i) { tc::mbar_init(BAR_FULL + 8 * i, 1); tc::mbar_init(BAR_EMPTY + 8 * i, WARPS); }
            abort_s = 0u;
            tc::fence_barrier_init();
        }
        __syncthreads();
    }
    if constexpr (!BASE) pdl_release();
    const uint8_t *w_packed = w.w_packed, *w_scale = w.w_scale;
    const uint16_t* x = w.x;
    if constexpr (BASE) {
        pdl_wait();
        w_packed = pdl_after(w_packed); w_scale = pdl_after(w_scale); x = pdl_after(x);
    }
    if (TMA && warp == WARPS) {
        if (lane == 0 && !SELFTEST) {
            uint32_t s = 0, ph = 0;
            for (uint32_t k0 = 0; k0 < p.K; k0 += DCM_KSTEP * WARPS) {          // (zero-filled past K and N)
                if (!tc::mbar_wait(BAR_EMPTY + 8 * s, ph ^ 1u, abort_flag, STATUS_WAIT_EXPIRED_PRODUCER)) break;
                const uint32_t st = ring + s * R::STAGE;
                tc::mbar_arrive_expect_tx(BAR_FULL + 8 * s, R::CODES + R::SCALES);
                for (uint32_t b = 0; b < uint32_t(R::BOXES); ++b)
                    tc::tma_load_2d(st + b * (R::ROWS * 128), &map_w, int32_t(k0 / 2 + 128 * b), int32_t(f0), BAR_FULL + 8 * s);
                tc::tma_load_2d(st + R::CODES, &map_s, int32_t(k0 / 16), int32_t(f0), BAR_FULL + 8 * s);
                if (++s == uint32_t(R::STAGES)) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    }

    if (!BASE && tid < DCM_MAX_TOKENS) {
        int32_t s = -1;
        if (p.seq_slot && tid < p.M) {
            s = p.seq_slot[tid];
            if (s >= 0) {
                if (uint32_t(s) >= p.max_loras) { record_status(STATUS_SLOT_OUT_OF_RANGE); s = -1; }
                else {
                    b_s[tid] = p.b_table[s];
                    rank_s[tid] = p.rank_table ? min(p.rank_table[s], p.max_rank) : p.max_rank;
                    if (p.a_table[s] == 0ull || b_s[tid] == 0ull) s = -1;
                }
            }
        }
        slot_s[tid] = s;
    }

    // ---- base: this thread's 32 codes per step of feature rows g and g + 8 of every tile, and of x rows g (+ 8 per n-tile) ----
    const uint32_t n_steps = (p.K + DCM_KSTEP - 1) / DCM_KSTEP;
    const uint8_t* code_row[TILES][2];
    const uint8_t* scale_row[TILES][2];
#pragma unroll
    for (int i = 0; i < TILES; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t f = min(f0 + 16 * i + 8 * h + g, p.N - 1u);          // (rows past N repeat the last one and are not stored)
            code_row[i][h] = w_packed + size_t(f) * (p.K / 2u) + 16 * t;
            scale_row[i][h] = w_scale + size_t(f) * (p.K / 16u) + 2 * t;
        }
    const uint16_t* x_row[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) x_row[n] = x + size_t(min(8 * n + g, p.M - 1u)) * w.x_row_stride + 32 * t;

    float acc[SETS][TILES][NT][4] = {};                                // sums `warp`, `warp` + WARPS
    // (one n-tile: x travels with the codes; more of them would not fit in registers and are read where they are used)
    constexpr bool X_AHEAD = NT == 1;
    uint4 xv[2][X_AHEAD ? 4 : 1];
    uint4 code[2][TILES][2];
    uint32_t sc[2][TILES][2];
    auto load = [&](uint32_t step, uint4 (&c)[TILES][2], uint32_t (&s)[TILES][2], uint4 (&xs)[X_AHEAD ? 4 : 1]) {
        const bool in = step * DCM_KSTEP + 32 * t < p.K;                        // (K is a multiple of 32)
#pragma unroll
        for (int i = 0; i < TILES; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                c[i][h] = in ? __ldcs(reinterpret_cast<const uint4*>(code_row[i][h] + step * (DCM_KSTEP / 2))) : make_uint4(0u, 0u, 0u, 0u);
                s[i][h] = in ? uint32_t(__ldg(reinterpret_cast<const uint16_t*>(scale_row[i][h] + step * (DCM_KSTEP / 16)))) : 0u;
            }
        if constexpr (X_AHEAD)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                xs[u] = in && g < p.M ? __ldg(reinterpret_cast<const uint4*>(x_row[0] + step * DCM_KSTEP + 8 * u)) : make_uint4(0u, 0u, 0u, 0u);
    };
    auto multiply = [&](uint32_t step, const uint4 (&c)[TILES][2], const uint32_t (&s)[TILES][2], const uint4 (&xs)[X_AHEAD ? 4 : 1],
                        float (&sum)[TILES][NT][4]) {
        const bool in = step * DCM_KSTEP + 32 * t < p.K;
        uint32_t mul[TILES][2][2];
#pragma unroll
        for (int i = 0; i < TILES; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) e4m3x2_to_bf16x2_shifted(e4m3x4_clear_nan(s[i][h]), 0x4140u, mul[i][h][0], mul[i][h][1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {                                           // eight K elements per thread at a time
            uint32_t xb[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                uint4 v;
                if constexpr (X_AHEAD) v = xs[u];
                else v = in && 8 * n + g < p.M ? __ldg(reinterpret_cast<const uint4*>(x_row[n] + step * DCM_KSTEP + 8 * u)) : make_uint4(0u, 0u, 0u, 0u);
                xb[n][0] = __byte_perm(v.x, v.z, 0x5410); xb[n][1] = __byte_perm(v.x, v.z, 0x7632);
                xb[n][2] = __byte_perm(v.y, v.w, 0x5410); xb[n][3] = __byte_perm(v.y, v.w, 0x7632);
            }
#pragma unroll
            for (int i = 0; i < TILES; ++i) {
                uint32_t a[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t word = u == 0 ? c[i][h].x : (u == 1 ? c[i][h].y : (u == 2 ? c[i][h].z : c[i][h].w));
                    e2m1x8_to_pairs(word, mul[i][h][u < 2 ? 0 : 1], a[h]);
                }
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    mma_bf16_16816(sum[i][n], a[0][0], a[1][0], a[0][1], a[1][1], xb[n][0], xb[n][1]);
                    mma_bf16_16816(sum[i][n], a[0][2], a[1][2], a[0][3], a[1][3], xb[n][2], xb[n][3]);
                }
            }
        }
    };
    if constexpr (TMA) {
        auto load_x = [&](uint32_t step, uint4 (&xs)[X_AHEAD ? 4 : 1]) {
            if constexpr (X_AHEAD) {
                const bool in = step < n_steps && g < p.M;
#pragma unroll
                for (int u = 0; u < 4; ++u) xs[u] = in ? __ldg(reinterpret_cast<const uint4*>(x_row[0] + step * DCM_KSTEP + 8 * u)) : make_uint4(0u, 0u, 0u, 0u);
            }
        };
        // a stage's chunk 4 (warp % 2) + t of box warp / 2, and bytes 8 warp + 2 t of its scale rows
        const uint32_t code_at = (warp >> 1) * (R::ROWS * 128) + g * 128 + (((4 * (warp & 1u) + t) ^ g) << 4);
        const uint32_t swz = WARPS == 8 ? (g >> 1) & 3u : (g >> 2) & 1u;
        const uint32_t scale_at = R::CODES + g * (8 * WARPS) + (((warp >> 1) ^ swz) << 4) + (warp & 1u) * 8 + 2 * t;
        uint32_t s = 0, ph = 0;
        auto turn = [&](uint32_t step, const uint4 (&xs)[X_AHEAD ? 4 : 1], float (&sum)[TILES][NT][4]) -> bool {
            // (a vote: lanes that gave up one by one would leave the others in warp-wide instructions, waiting for them)
            if (!tc::mbar_wait_warp(BAR_FULL + 8 * s, ph, abort_flag, STATUS_WAIT_EXPIRED_DEQUANT)) return false;
            const uint32_t st = ring + s * R::STAGE;
#pragma unroll
            for (int i = 0; i < TILES; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    code[0][i][h] = tc::lds128(st + code_at + (16 * i + 8 * h) * 128);
                    uint16_t v;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(st + scale_at + (16 * i + 8 * h) * (8 * WARPS)));
                    sc[0][i][h] = v;
                }
            if (step < n_steps) multiply(step, code[0], sc[0], xs, sum);
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(BAR_EMPTY + 8 * s);
            if (++s == uint32_t(R::STAGES)) { s = 0; ph ^= 1u; }
            return true;
        };
        if (warp < WARPS) {
            load_x(warp, xv[0]);
            for (uint32_t step = warp; step - warp < n_steps; step += 2 * WARPS) {      // (all warps go through all stages)
                load_x(step + WARPS, xv[1]);
                if (!turn(step, xv[0], acc[0]) || step + WARPS - warp >= n_steps) break;
                load_x(step + 2 * WARPS, xv[0]);
                if (!turn(step + WARPS, xv[1], acc[SETS - 1])) break;
            }
        }
    } else {
        load(warp, code[0], sc[0], xv[0]);
        for (uint32_t step = warp; step < n_steps; step += 2 * WARPS) {
            load(step + WARPS, code[1], sc[1], xv[1]);
            multiply(step, code[0], sc[0], xv[0], acc[0]);
            load(step + 2 * WARPS, code[0], sc[0], xv[0]);
            if (step + WARPS < n_steps) multiply(step + WARPS, code[1], sc[1], xv[1], acc[SETS - 1]);
        }
    }

    if constexpr (BASE) pdl_release();
    // ---- LoRA granules of this warp ----
    if (!BASE && p.seq_slot) {
        __syncthreads();                                                        // slot_s, rank_s, b_s
        // this CTA's rows of B into L2 while the shrink may still run
        for (uint32_t m = warp; (!TMA || warp < WARPS) && m < p.M; m += WARPS) {
            if (slot_s[m] < 0 || lane >= TILES * 16u || f0 + lane >= p.N) continue;
            const uint64_t row = b_s[m] + size_t(f0 + lane) * p.max_rank * 2u;
            for (uint32_t j = 0; j < rank_s[m]; j += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"((row + 2u * j) & ~15ull));
        }
        if (p.wait_for_shrink) pdl_wait();
        // slots of the token this thread loads t for, and of the two tokens (columns) whose sums it holds
        int32_t own[NT], col[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            own[n] = slot_s[8 * n + g];
            col[n][0] = slot_s[8 * n + 2 * t];
            col[n][1] = slot_s[8 * n + 2 * t + 1];
        }
        const int32_t lane_slot = lane < DCM_MAX_TOKENS ? slot_s[lane] : -1;
        for (uint32_t left = __ballot_sync(0xFFFFFFFFu, lane_slot >= 0); left;) {
            const uint32_t first = __ffs(left) - 1;                             // first token of this slot
            const int32_t s = __shfl_sync(0xFFFFFFFFu, lane_slot, first);
            left &= ~__ballot_sync(0xFFFFFFFFu, lane_slot == s);
            const uint32_t rank = rank_s[first];
            const uint16_t* B = reinterpret_cast<const uint16_t*>(b_s[first]);
            const bool b_vec = (reinterpret_cast<uintptr_t>(B) & 7u) == 0u;
            for (uint32_t j = 0; 16 * j < rank; ++j) {
                const uint32_t to = (uint32_t(s) + 3u * j) % DCM_SUMS;
                if (to % WARPS != warp) continue;
                const uint32_t j0 = 16 * j + 4 * t;
                const bool in = j0 < p.max_rank;                                // (max_rank is a multiple of 8)
                uint2 tv[NT];
#pragma unroll
                for (int n = 0; n < NT; ++n)
                    tv[n] = in && own[n] == s ? *reinterpret_cast<const uint2*>(p.t + size_t(8 * n + g) * p.max_rank + j0) : make_uint2(0u, 0u);
#pragma unroll
                for (int i = 0; i < TILES; ++i) {
                    uint2 bv[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint16_t* q = B + size_t(min(f0 + 16 * i + 8 * h + g, p.N - 1u)) * p.max_rank + j0;
                        if (!in) bv[h] = make_uint2(0u, 0u);
                        else if (b_vec) bv[h] = __ldg(reinterpret_cast<const uint2*>(q));
                        else bv[h] = make_uint2(uint32_t(q[0]) | uint32_t(q[1]) << 16, uint32_t(q[2]) | uint32_t(q[3]) << 16);
                    }
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        // into the columns of this slot alone: an infinity in one adapter's B, times the zeros that stand for
                        // the other tokens, must not reach them
                        float d[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) d[e] = SETS > 1 && to >= WARPS ? acc[SETS - 1][i][n][e] : acc[0][i][n][e];
                        mma_bf16_16816(d, bv[0].x, bv[1].x, bv[0].y, bv[1].y, tv[n].x, tv[n].y);
#pragma unroll
                        for (int h = 0; h < SETS; ++h)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[h][i][n][e] = col[n][e & 1] == s && to / WARPS == h ? d[e] : acc[h][i][n][e];
                    }
                }
            }
        }
    }

    // ---- the partial sums, added in their order ----
    if (!TMA || warp < WARPS)
#pragma unroll
    for (int h = 0; h < SETS; ++h)
#pragma unroll
        for (int i = 0; i < TILES; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) part[warp + h * WARPS][8 * n + 2 * t + (e & 1)][16 * i + g + 8 * (e >> 1)] = acc[h][i][n][e];
    __syncthreads();
    // (a tile whose weights did not all arrive stays unwritten)
    const bool whole_sums = !TMA || (warp < WARPS && !*abort_flag);
    for (uint32_t i = tid; whole_sums && i < NT * 8 * TILES * 16; i += (32 * WARPS)) {          // (whole warps: a multiple of 128)
        const uint32_t m = i / (TILES * 16), fi = i % (TILES * 16), f = f0 + fi;
        float sum = part[0][m][fi];
#pragma unroll
        for (int k = 1; k < DCM_SUMS; ++k) sum += part[k][m][fi];
        const uint32_t bits = f32_to_bf16_bits(sum * p.out_scale);
        const bool in = m < p.M && f < p.N;
        const size_t at = size_t(m) * p.out_row_stride + p.y_col0 + f;
        if (p.n_dest == 1) {
            if (in) p.y_dest[0][at] = uint16_t(bits);
            continue;
        }
        // several buffers, peers' among them (their rows allow 16-byte stores): eight lanes' features in one store.  (Into one
        // buffer the shuffles cost more than the narrow stores: a decode layer 97.6 instead of 96.7 us.)
        const uint32_t w0 = bits | __shfl_down_sync(0xFFFFFFFFu, bits, 1) << 16, w1 = __shfl_down_sync(0xFFFFFFFFu, w0, 2);
        const uint32_t w2 = __shfl_down_sync(0xFFFFFFFFu, w0, 4), w3 = __shfl_down_sync(0xFFFFFFFFu, w1, 4);
        if (!in) continue;
        const bool whole = (f & ~7u) + 8u <= p.N;
        for (uint32_t r = 0; r < p.n_dest; ++r) {
            if (!whole) p.y_dest[r][at] = uint16_t(bits);
            else if (lane % 8u == 0) *reinterpret_cast<uint4*>(p.y_dest[r] + at) = make_uint4(w0, w1, w2, w3);
        }
    }
    if constexpr (TMA)
        if (*abort_flag) {
            // give copies that may still be in flight time to land before shared memory is released
            const uint64_t t0 = tc::global_timer_ns();
            while (tc::global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
}

}  // namespace atlas
