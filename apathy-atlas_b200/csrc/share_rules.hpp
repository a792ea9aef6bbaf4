// Who takes what: index rules that involve neither memory nor a device, in plain C++ so that they are checked on the CPU.
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define ATLAS_HD __host__ __device__
#else
#define ATLAS_HD
#endif

namespace atlas {

// Granules are dealt out in blocks of four: of `ks` CTAs, CTA kz takes the blocks kz, kz + ks, ...  The granule that follows `g`
// among one CTA's, whose first is 4 kz.
ATLAS_HD constexpr uint32_t next_own_granule(uint32_t g, uint32_t ks) { return (g & 3u) != 3u ? g + 1u : g + 4u * ks - 3u; }

// The grid of the mma.sync shrink: `slots` slots of `granules` granules over `chunks` chunks of `rows` rows.
struct MmaShrinkGrid {
    uint32_t ksplit;              // CTAs of a cluster, sharing K
    uint32_t row_parts_log2;      // 2^this clusters share a slot's rows
    uint32_t prefetch_ctas;       // the first CTAs, which are resident while the kernel ahead still runs: they prefetch A
};
// what of the machine a dependent wants while this grid runs (tiles: all of it, for one tile of 128 features a CTA; all: for longer)
enum class MachineBeside { none, part, all, tiles };
constexpr uint32_t MMA_SHRINK_KSPLIT = 8, MMA_SHRINK_PASS = 32, MMA_SHRINK_CTAS_PER_SM = 8;
inline MmaShrinkGrid mma_shrink_grid(uint32_t slots, uint32_t granules, uint32_t chunks, uint32_t rows, uint32_t sm_count, MachineBeside wanted_beside) {
    const uint64_t items = uint64_t(slots) * granules * chunks;
    // K split: eight for the sake of loads in flight; fewer where the dependent kernel runs beside this grid on a part of the machine
    // only (a decode batch) and this grid would otherwise be so large that the dependent's CTAs find no room until it has drained.
    const uint64_t half = uint64_t(sm_count) * (MMA_SHRINK_CTAS_PER_SM / 2);
    MmaShrinkGrid g{MMA_SHRINK_KSPLIT, 0, 0};
    while (wanted_beside == MachineBeside::part && g.ksplit > 2 && items * g.ksplit > half) g.ksplit >>= 1;
    // Clusters sharing the rows of each, up to one per 32 rows that a slot may have.  Beside a dependent that wants the whole machine CTAs
    // without rows are not free: no more than half of what can be resident is taken then, unless the rows of an average slot fill them or
    // the batch has one chunk (two, for two clusters).  One / more (us), CTAs in parentheses: 160 tokens, 2 adapters of rank 16 x 4096 x
    // 4096 34.4 (16) / 21.8 (128), 32 of rank 32 in sequences 28.3 (512) / 24.3 (1024); 512 tokens, 8 of rank 64 in sequences 48.3 (512)
    // / 40.6 (1024); 8 of rank 16, mixed 30.0 (128) / 26.1 (512) / 33.4 (1024), x 14336 60 / 54 / 75; 1000 tokens, 16 of rank 16, mixed
    // 42.4 (512) / 44.1 (1024); beside 1024 features, 512 tokens, 128 of rank 16 42.0 (512) / 32.4 (1024), 64 tokens with an adapter of
    // rank 64 each 36.0 / 36.1; with nothing beside it, 1000 tokens, 8 of rank 16 in sequences 62.7 (512) / 58.2 (1024).
    // A second cluster to rows that fill it comes before everything being resident beside a kernel of one tile a CTA (1024 / 2048):
    // 1000 tokens, 8 of rank 64 in sequences x 4096 x 4096 63.5 / 51.1, x 14336 166.5 / 133.0, mixed 50.2 / 49.0 and 126.0 / 121.1; but
    // beside the persistent kernel (14336 x 4096, 700 tokens, mixed) 86.4 / 93.0.
    auto bound = [&](uint32_t log2) {
        const bool filled = rows >= (uint64_t(slots) * MMA_SHRINK_PASS << log2) || chunks == 1 || (chunks == 2 && log2 == 0);
        if (wanted_beside == MachineBeside::tiles && filled && log2 == 0) return 4 * half;
        return (wanted_beside == MachineBeside::all || wanted_beside == MachineBeside::tiles) && !filled ? half : 2 * half;
    };
    while ((MMA_SHRINK_PASS << g.row_parts_log2) < rows && (items * g.ksplit << (g.row_parts_log2 + 1)) <= bound(g.row_parts_log2)) ++g.row_parts_log2;
    g.prefetch_ctas = sm_count * MMA_SHRINK_CTAS_PER_SM;
    return g;
}

}  // namespace atlas
