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

}  // namespace atlas
