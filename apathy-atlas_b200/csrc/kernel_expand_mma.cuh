// Staged expand + fold on the tensor cores, the arithmetic of lora_expand_fold_kernel (kernels_simt.cuh):
//   delta = bf16(sum_j xa[m,j] * B_s[o,j]);  out[m,o] = bf16(f32(out[m,o]) + scale_s * f32(delta)),  s = the row's slot.
//
// What it cannot do without is reading and writing `out` once; the CUDA-core form reads a B row per thread and row and an xa
// element per FMA, which made it 321 us at 2048 x 4096, rank 64 (33.6 MB of `out`: 5 us at the copy rate).
//
// A CTA owns 128 features (32 per warp) and up to 128 rows.  It sorts its rows by slot, so that sixteen consecutive rows
// (the M of mma.sync.m16n8k16) hold few runs of one slot, and takes the runs in turn: B_s fragments stay in registers for as
// long as the slot does not change, the next run's rows are on their way, the product of a run starts from zero and is folded
// into the run's rows alone.  (Rows of other slots in the same sixteen are computed and dropped, not masked with zeros: an
// infinity in one adapter's B must not reach another adapter's rows.)  A decode batch has few rows and as many runs as
// adapters, each waiting for its B_s: `splits` CTAs share the runs of a chunk.
//
// Fragments: in every 16-wide K step the thread of quad lane t holds ranks 4t..4t+3 of xa rows g, g+8 and of its B row (64-bit
// loads; both operands use the same assignment, so each rank meets its partner).  The four n-tiles of a warp interleave
// their columns (column c of tile i = feature 8 (c / 2) + 2 i + c % 2), so that a thread ends up with eight consecutive
// features of its rows and `out` moves in 128-bit accesses.
#pragma once

#include "kernel_shrink_mma.cuh"

namespace atlas {

constexpr int EXM_THREADS = 128;
constexpr int EXM_ROWS = 128;        // rows of a chunk: one per thread while they are sorted
constexpr int EXM_OUTS = 128;        // features per CTA
constexpr int EXM_MAX_RANK = 128;    // B_s fragments of 32 features are held in registers: 64 at this rank

// KS: 16-wide K steps held in registers, >= ceil(max_rank / 16); CTAS on an SM
template <int KS, int CTAS = KS >= 8 ? 3 : (KS >= 4 ? 4 : 5)>
__global__ void __launch_bounds__(EXM_THREADS, CTAS)
lora_expand_mma_kernel(ExpandParams p, uint32_t chunk, uint32_t splits) {
    constexpr bool AHEAD = KS <= 4;                          // xa too (more of it does not fit beside B_s)
    __shared__ __align__(16) uint32_t slot_in[EXM_ROWS];     // slot, ~0 for a row without a term
    __shared__ int32_t slot_s[EXM_ROWS];
    __shared__ uint64_t b_s[EXM_ROWS];
    __shared__ float scale_s[EXM_ROWS];
    __shared__ uint16_t row_s[EXM_ROWS];
    __shared__ uint16_t run_s[EXM_ROWS + 1];                 // first row of every run, then the end
    __shared__ uint32_t warp_runs[EXM_THREADS / 32];
    pdl_release();
    pdl_wait();
    p.b_uniform = pdl_after(p.b_uniform); p.b_table = pdl_after(p.b_table); p.scale_table = pdl_after(p.scale_table); p.xa = pdl_after(p.xa);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t m0 = (blockIdx.y / splits) * chunk, split = blockIdx.y % splits;
    const uint32_t n_in = min(chunk, p.M - m0);

    // ---- this chunk's rows that take a term, sorted by slot, and their runs: of one slot, within sixteen rows ----
    uint32_t n, n_runs = 0;
    {
        int32_t s = -1;
        uint64_t b_addr = reinterpret_cast<uint64_t>(p.b_uniform);
        float scale = p.scale_uniform;
        if (tid < n_in) {
            s = p.seq_slot ? p.seq_slot[m0 + tid] : 0;
            if (p.seq_slot && s >= 0) {
                if (uint32_t(s) >= p.max_loras) { record_status(STATUS_SLOT_OUT_OF_RANGE); s = -1; }
                else {
                    b_addr = p.b_table[s];
                    scale = p.scale_table[s];
                    if (b_addr == 0ull || (p.a_table && p.a_table[s] == 0ull)) s = -1;
                }
            }
        }
        slot_in[tid] = uint32_t(s);
        n = __syncthreads_count(s >= 0);
        if (s >= 0) {
            uint32_t pos = p.seq_slot ? 0u : tid;             // (one adapter for all rows: sorted already)
            for (uint32_t i = 0; p.seq_slot && i < n_in; i += 4) {
                const uint4 o = *reinterpret_cast<const uint4*>(&slot_in[i]);          // (~0 is larger than any slot)
                pos += (o.x < uint32_t(s) || (o.x == uint32_t(s) && i < tid)) + (o.y < uint32_t(s) || (o.y == uint32_t(s) && i + 1 < tid)) +
                       (o.z < uint32_t(s) || (o.z == uint32_t(s) && i + 2 < tid)) + (o.w < uint32_t(s) || (o.w == uint32_t(s) && i + 3 < tid));
            }
            slot_s[pos] = s;
            b_s[pos] = b_addr;
            scale_s[pos] = scale;
            row_s[pos] = uint16_t(tid);
        }
        __syncthreads();
        const bool starts = tid < n && (tid % 16u == 0u || slot_s[tid] != slot_s[tid - 1u]);
        const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, starts);
        if (lane == 0) warp_runs[warp] = __popc(ballot);
        __syncthreads();
        uint32_t at = __popc(ballot & ((1u << lane) - 1u));
#pragma unroll
        for (uint32_t w = 0; w < EXM_THREADS / 32; ++w) {
            if (w < warp) at += warp_runs[w];
            n_runs += warp_runs[w];
        }
        if (starts) run_s[at] = uint16_t(tid);
        if (tid == 0) run_s[n_runs] = uint16_t(n);
        __syncthreads();
    }
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint32_t o0 = blockIdx.x * EXM_OUTS + warp * 32;            // this warp's 32 features
    if (o0 >= p.n_out) return;
    const uint32_t o = o0 + 8 * t;                                     // this thread's eight
    const uint32_t ks_n = (p.max_rank + 15u) / 16u;
    const bool whole = o + 8u <= p.n_out;
    const bool vec = whole && p.out_row_stride % 8u == 0u && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0u;

    uint2 b[KS][4];
    int32_t b_slot = -1;
    float scale = 0.0f;
    // What a run reads of `out` and xa is requested one run ahead: with one run at a time a CTA was a chain of as many latencies as it
    // has runs (base, shrink and this: 2048 tokens x 4096 x 4096, rank 64 88.7 -> 79.3 us; 128 x 8192 x 2048, 64 adapters of rank 128
    // 110.8 -> 99.6).
    struct Rows {
        uint32_t m[2];
        bool in_run[2];
        uint4 old[2];
        uint2 a[AHEAD ? KS : 1][2];
    };
    auto load_xa = [&](const Rows& r, int k, int h) {
        const uint32_t j = 16 * k + 4 * t;
        return j < p.max_rank ? *reinterpret_cast<const uint2*>(p.xa + size_t(r.m[h]) * p.max_rank + j) : make_uint2(0u, 0u);
    };
    auto request = [&](uint32_t run, Rows& r) {
        const uint32_t lo = run_s[run], hi = run_s[run + 1];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // rows g and g + 8 of the sixteen, where they belong to the run
            const uint32_t i = (lo & ~15u) + g + 8 * h;
            r.in_run[h] = i >= lo && i < hi;
            r.m[h] = m0 + row_s[r.in_run[h] ? i : lo];
            r.old[h] = make_uint4(0u, 0u, 0u, 0u);
            if (r.in_run[h] && vec) r.old[h] = *reinterpret_cast<const uint4*>(p.out + size_t(r.m[h]) * p.out_row_stride + o);
        }
        if constexpr (AHEAD)
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) r.a[k][h] = load_xa(r, k, h);
    };
    Rows next;
    if (split < n_runs) request(split, next);
    for (uint32_t run = split; run < n_runs; run += splits) {          // (every `splits`-th run is this CTA's)
        const Rows r = next;
        const uint32_t run_lo = run_s[run];
        const int32_t s = slot_s[run_lo];
        const auto& m = r.m;
        const auto& in_run = r.in_run;
        const auto& old = r.old;
        if (run + splits < n_runs) request(run + splits, next);
        if (s != b_slot) {
            b_slot = s;
            const uint16_t* B = reinterpret_cast<const uint16_t*>(b_s[run_lo]);
            scale = scale_s[run_lo];
            const bool b_vec = (reinterpret_cast<uintptr_t>(B) & 7u) == 0u;
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t f = o0 + 8 * (g >> 1) + 2 * i + (g & 1u), j = 16 * k + 4 * t;
                    b[k][i] = make_uint2(0u, 0u);
                    if (f < p.n_out && j < p.max_rank) {            // (max_rank is a multiple of 8: four ranks are inside or out)
                        const uint16_t* q = B + size_t(f) * p.max_rank + j;
                        if (b_vec) b[k][i] = __ldg(reinterpret_cast<const uint2*>(q));
                        else b[k][i] = make_uint2(uint32_t(q[0]) | uint32_t(q[1]) << 16, uint32_t(q[2]) | uint32_t(q[3]) << 16);
                    }
                }
        }
        float acc[4][4] = {};
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            if (uint32_t(k) < ks_n) {
                uint2 a[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if constexpr (AHEAD) a[h] = r.a[k][h];
                    else a[h] = load_xa(r, k, h);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_bf16_16816(acc[i], a[0].x, a[1].x, a[0].y, a[1].y, b[k][i].x, b[k][i].y);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!in_run[h]) continue;
            uint16_t* dst = p.out + size_t(m[h]) * p.out_row_stride + o;
            uint32_t d[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] = pack_bf16x2(acc[i][2 * h], acc[i][2 * h + 1]);
            if (vec) {
                const uint32_t base[4] = {old[h].x, old[h].y, old[h].z, old[h].w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[i] = pack_bf16x2(__fadd_rn(bf16_lo(base[i]), __fmul_rn(scale, bf16_lo(d[i]))),
                                       __fadd_rn(bf16_hi(base[i]), __fmul_rn(scale, bf16_hi(d[i]))));
                *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (o + e < p.n_out) {
                        const float delta = (e & 1) ? bf16_hi(d[e >> 1]) : bf16_lo(d[e >> 1]);
                        dst[e] = f32_to_bf16_bits(__fadd_rn(__uint_as_float(uint32_t(dst[e]) << 16), __fmul_rn(scale, delta)));
                    }
            }
            if (p.delta_out && whole && p.n_out % 8u == 0u && (reinterpret_cast<uintptr_t>(p.delta_out) & 15u) == 0u) {
                *reinterpret_cast<uint4*>(p.delta_out + size_t(m[h]) * p.n_out + o) = make_uint4(d[0], d[1], d[2], d[3]);
            } else if (p.delta_out) {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (o + e < p.n_out) p.delta_out[size_t(m[h]) * p.n_out + o + e] = uint16_t(d[e >> 1] >> (16 * (e & 1)));
            }
        }
    }
}

}  // namespace atlas
