// C ABI of the B200 NVFP4 + multi-LoRA linear path: argument validation, variant dispatch and
// kernel launches.  Single translation unit (the kernels share one device status word).
//
// Host-side operator layer (namespace atlas::ops) mirrors the reference's launch wrappers:
//   ops::apply_lora_bgmv   <- crates/spark-model/src/layers/ops/lora_delta.rs:269-314
//   ops::apply_lora_delta  <- crates/spark-model/src/layers/ops/lora_delta.rs:145-235
//   ops::w4a16_gemm        <- crates/spark-model/src/layers/ops/gemm_dense.rs:258-281
//   ops::nvfp4_lora_linear    (fused; new)
// Like them it only launches: no allocation, no synchronisation, no host read of device data.
#include "atlas_b200.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>

#include "common.cuh"
#include "kernel_tc.cuh"
#include "kernel_tc_persist.cuh"
#include "kernel_decode_mma.cuh"
#include "kernel_dense_tc.cuh"
#include "kernels_simt.cuh"
#include "kernel_shrink_mma.cuh"
#include "kernel_expand_mma.cuh"
#include "kernel_shrink_tc.cuh"
#include "kernels_mlp_glue.cuh"
#include "kernel_push.cuh"
#include "kernel_kv_epilogue.cuh"

namespace atlas {

static thread_local int t_last_variant = ATLAS_B200_VARIANT_NONE;
static thread_local uint32_t t_last_shape[8] = {0, 0, 0, 0, 0, 0, 0, 0};
static unsigned long long* g_profile_buf = nullptr;   // device buffer for per-CTA cycle counters (diagnostics)
static size_t g_profile_words = 0;

static inline int cuda_status(cudaError_t e) { return e == cudaSuccess ? ATLAS_B200_OK : ATLAS_B200_ERR_CUDA_BASE - int(e); }
static inline int launch_status() { return cuda_status(cudaGetLastError()); }
// A launch of a kernel that begins with pdl_wait(): it may start while its predecessor in the stream finishes.
template <typename... P, typename... A>
static int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}
static inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// ---------------------------------------------------------------------------------------------
// device capability and the tensor-map encoder (resolved from the driver at first use; the
// library does not link libcuda)
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// What the launcher learns about a device and the per-device settings it has applied.  Function attributes
// (opt-in shared memory, carve-out) and occupancy answers belong to a device, so everything here is kept per
// device ordinal and created under a lock the first time that device is current in a call.
constexpr int kMaxDevices = 64;
constexpr int kPersistKernels = 5;
struct DeviceState {
    std::atomic<bool> ready{false};
    bool sm100 = false;
    int sm_count = 148;
    bool tc_attr_set[60] = {};        // token tiles 16..256 x {A16, A4} x {single CTA, CTA pair} x {K of whole raw stages, not, ranks above 64}
    int known_clusters[20][9] = {};   // resident clusters per kernel instance and K split; 0 = not asked yet
    bool persist_attr_set[kPersistKernels] = {};
    int persist_clusters[kPersistKernels] = {};
    bool carveout_set = false;
    bool shrink_tc_attr_set = false;
    int shrink_tc_clusters[SHT_MAX_KSPLIT + 1] = {};   // resident clusters of that many CTAs of the prefill shrink; 0 = not asked yet
    bool push_attr_set = false;
    bool dense_attr_set[5] = {};      // token tiles 16, 32, 64, 128, 256 of the dense-BF16 kernel
    bool decode_attr_set[8] = {};     // TMA form of the small-batch kernel: features of a CTA x {four, eight warps} x {adapters, none}
};
static DeviceState g_dev[kMaxDevices];
static std::mutex g_dev_mutex;
static EncodeTiledFn g_encode = nullptr;

// state of the current device; nullptr when there is none (no driver, ordinal out of range)
static DeviceState* device_state() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { (void)cudaGetLastError(); return nullptr; }
    DeviceState& st = g_dev[dev];
    if (st.ready.load(std::memory_order_acquire)) return &st;
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    if (!st.ready.load(std::memory_order_relaxed)) {
        int major = 0;
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
        st.sm100 = (major == 10);
        cudaDeviceGetAttribute(&st.sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (st.sm_count <= 0) st.sm_count = 148;
        if (!g_encode) {
            void* fn = nullptr;
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess)
                g_encode = reinterpret_cast<EncodeTiledFn>(fn);
        }
        st.ready.store(true, std::memory_order_release);
    }
    return &st;
}

static int rt_sm_count() { DeviceState* st = device_state(); return st ? st->sm_count : 148; }

// Encoded tensor maps are a pure function of (address, shape, strides, box, type, swizzle): a serving loop calls with the
// same tensors step after step, so recent encodings are kept per host thread and a repeated call costs a compare instead of a
// driver call per map.  A 32-layer model has some 1300 maps per batch shape (some 1500 with adapters of rank 32 or 64, whose B
// is fetched in boxes of two widths; 450 where the smallest batches have their weights by TMA): 4096 are held, in sets of four of which the least
// recently used one is replaced (1 MiB per calling thread, allocated at its first call and given back when the thread ends; with
// no memory for it every map is encoded anew).  With 64 entries a decode step of one layer evicted its own maps and spent about
// half of its host time (145 us) in the driver's encoder.
struct MapKey {
    const void* base;
    uint64_t dims[3], strides[2];
    uint32_t box[3];
    int32_t rank, dtype, swizzle;
};
struct MapEntry {
    MapKey key;
    uint64_t used;           // t_map_tick at its last use; 0 = empty
    CUtensorMap map;
};
static_assert(sizeof(MapEntry) == 256, "4096 entries are 1 MiB");
constexpr uint32_t kMapSets = 1024, kMapWays = 4;
static thread_local std::unique_ptr<MapEntry[]> t_map_cache;
static thread_local uint64_t t_map_tick = 0;

static bool encode_tiled(CUtensorMap* map, CUtensorMapDataType dt, uint32_t rank, const void* base, const uint64_t* dims,
                         const uint64_t* strides, const uint32_t* box, CUtensorMapSwizzle swz,
                         CUtensorMapL2promotion promo = CU_TENSOR_MAP_L2_PROMOTION_L2_128B) {
    MapKey key;
    std::memset(&key, 0, sizeof(key));
    key.base = base; key.rank = int32_t(rank); key.dtype = int32_t(dt); key.swizzle = int32_t(swz) | (int32_t(promo) << 8);
    for (uint32_t i = 0; i < rank; ++i) { key.dims[i] = dims[i]; key.box[i] = box[i]; }
    for (uint32_t i = 0; i + 1 < rank; ++i) key.strides[i] = strides[i];
    uint64_t h = reinterpret_cast<uintptr_t>(base) * 0x9E3779B97F4A7C15ull;
    h ^= (key.dims[0] * 31 + key.dims[1]) * 0xBF58476D1CE4E5B9ull + key.box[0] * 131 + key.box[1] * 17 + uint64_t(key.swizzle);
    h ^= uint64_t(key.rank) * 0x94D049BB133111EBull + key.dims[2] + key.strides[0] * 0x2545F4914F6CDD1Dull;
    h *= 0x9E3779B97F4A7C15ull;
    if (!t_map_cache) t_map_cache.reset(new (std::nothrow) MapEntry[size_t(kMapSets) * kMapWays]());
    MapEntry* e = nullptr;                                   // the set's least recently used entry
    if (t_map_cache) {
        MapEntry* set = e = &t_map_cache[size_t((h >> 32) % kMapSets) * kMapWays];
        for (uint32_t w = 0; w < kMapWays; ++w) {
            if (set[w].used && std::memcmp(&set[w].key, &key, sizeof(key)) == 0) {
                set[w].used = ++t_map_tick;
                *map = set[w].map;
                return true;
            }
            if (set[w].used < e->used) e = &set[w];
        }
    }
    cuuint64_t gd[3], gs[2];
    cuuint32_t bx[3], es[3] = {1, 1, 1};
    for (uint32_t i = 0; i < rank; ++i) { gd[i] = dims[i]; bx[i] = box[i]; }
    for (uint32_t i = 0; i + 1 < rank; ++i) gs[i] = strides[i];
    auto encode = [&] {
        return g_encode(map, dt, rank, const_cast<void*>(base), gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, promo,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult rc = encode();
    int dev = -1;
    // a thread whose first call of CUDA this is has no context yet, and unlike the runtime's calls this one does not make one current
    if ((rc == CUDA_ERROR_INVALID_CONTEXT || rc == CUDA_ERROR_NOT_INITIALIZED) && cudaGetDevice(&dev) == cudaSuccess &&
        cudaSetDevice(dev) == cudaSuccess)
        rc = encode();
    if (rc != CUDA_SUCCESS) return false;
    if (e) { e->key = key; e->map = *map; e->used = ++t_map_tick; }
    return true;
}

static bool encode_2d(CUtensorMap* map, CUtensorMapDataType dt, size_t elem, const void* base, uint64_t inner,
                      uint64_t outer, uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer,
                      CUtensorMapSwizzle swz, CUtensorMapL2promotion promo = CU_TENSOR_MAP_L2_PROMOTION_L2_128B) {
    (void)elem;
    const uint64_t dims[2] = {inner, outer}, strides[1] = {row_stride_bytes};
    const uint32_t box[2] = {box_inner, box_outer};
    return encode_tiled(map, dt, 2, base, dims, strides, box, swz, promo);
}

// ---------------------------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------------------------
namespace ops {

// tensor-core shrink where rows can be read with aligned 128-bit loads in whole 32-element chunks
static bool shrink_takes_mma_path(const ShrinkParams& p) {
    return (p.k_in % 32 == 0) && (p.x_row_stride % 8 == 0) && aligned(p.x, 16) && (p.seq_slot || aligned(p.a_uniform, 4));
}

// How many clusters of `ksplit` CTAs of the prefill shrink can be resident at once (they live inside one GPC: fewer than the SM
// count suggests).  Asked once per device.
static int shrink_tc_clusters(DeviceState& dst, uint32_t ksplit) {
    if (dst.shrink_tc_clusters[ksplit] == 0) {
        cudaLaunchConfig_t q{};
        q.gridDim = dim3(ksplit);
        q.blockDim = dim3(SHT_THREADS);
        q.dynamicSmemBytes = SHT_SMEM_BYTES;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ksplit;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        q.attrs = attr;
        q.numAttrs = 1;
        int n = 0;
        dst.shrink_tc_clusters[ksplit] = cudaOccupancyMaxActiveClusters(&n, lora_shrink_tc_kernel, &q) == cudaSuccess && n > 0 ? n : -1;
        (void)cudaGetLastError();
    }
    return dst.shrink_tc_clusters[ksplit];
}

// `beside`: what of the machine the kernel behind it wants, which is then released as soon as this one's CTAs run (none: not released)
static int launch_shrink(ShrinkParams p, uint32_t n_slots, cudaStream_t st, MachineBeside beside = MachineBeside::none) {
    const bool release_dependents = beside != MachineBeside::none;
    p.release_dependents = release_dependents ? 1u : 0u;
    p.profile = nullptr;
    if (p.M == 0 || p.max_rank == 0) return ATLAS_B200_OK;
    // Same shared-memory carve-out as the tcgen05 kernel, so that kernel's CTAs can become resident
    // next to this grid's instead of waiting for the SMs to drain and be reconfigured.
    DeviceState* dst = device_state();
    if (dst && !dst->carveout_set) {
        cudaFuncSetAttribute(lora_shrink_grouped_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        cudaFuncSetAttribute(lora_shrink_mma_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        dst->carveout_set = true;
    }
    const bool mma_ok = shrink_takes_mma_path(p);
    if (p.tile_out && !mma_ok) return ATLAS_B200_ERR_DIMS;      // tile output exists in the tensor-core shrink only
    const void* a_base = p.seq_slot ? p.a_pool_base : static_cast<const void*>(p.a_uniform);
    const size_t a_stride = p.seq_slot ? p.a_slot_stride : size_t(p.max_rank) * p.k_in * 2;
    if (mma_ok && p.M >= 1024 && !release_dependents && p.k_in % SHT_KSTAGE == 0 && p.max_rank % 16 == 0 && p.max_rank <= 256 &&
        n_slots <= 4096 && dst && dst->sm100 && g_encode && a_base && aligned(a_base, 16) && a_stride % 16 == 0 &&
        (!p.tile_out || (p.part_rows && p.chunk % p.part_rows == 0 && p.chunk >= uint32_t(SHT_ROWS)))) {
        // a prefill batch: one cluster per 128 tokens and all ranks of all their adapters on the tcgen05 tensor cores,
        // x read once (kernel_shrink_tc.cuh); its rows lie in at most two token tiles
        if (!dst->shrink_tc_attr_set) {
            cudaError_t e = cudaFuncSetAttribute(lora_shrink_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SHT_SMEM_BYTES);
            if (e != cudaSuccess) return cuda_status(e);
            dst->shrink_tc_attr_set = true;
        }
        CUtensorMap map_x, map_a;
        if (!encode_2d(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.x, p.k_in, p.M, uint64_t(p.x_row_stride) * 2, SHT_KSTAGE, SHT_ROWS,
                       CU_TENSOR_MAP_SWIZZLE_128B))
            return ATLAS_B200_ERR_DIMS;
        {
            const uint64_t dims[3] = {p.k_in, p.max_rank, p.seq_slot ? n_slots : 1u};
            const uint64_t strides[2] = {uint64_t(p.k_in) * 2, uint64_t(a_stride)};
            const uint32_t box[3] = {SHT_KSTAGE, p.max_rank, 1};
            if (!encode_tiled(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a_base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
                return ATLAS_B200_ERR_DIMS;
        }
        p.a_pool_base = nullptr;      // host-side fields: not part of what the kernel reads
        if (p.m_begin % 64 != 0 || p.m_begin >= p.M) return ATLAS_B200_ERR_DIMS;
        const uint32_t rows = p.m_count ? std::min(p.m_count, p.M - p.m_begin) : p.M - p.m_begin;
        // CTAs per 128 rows, each contracting a share of K: two, or four or eight where the clusters of the batch (the whole of it, not
        // this launch's range: a row's result must not depend on how the batch is cut into launches) are all resident at once — a
        // second wave costs more than the split gains (4352 tokens, 34 clusters of four: 36 instead of 29 us).  Two / four / eight CTAs,
        // eight adapters of rank 64: 1237 tokens, K = 4096 34 / 25 / 22 us, K = 14336 81 / 48 / 34 us; 4096 tokens 29 / 22 and 68 / 43 us.
        const uint32_t k_blocks = p.k_in / SHT_KSTAGE, row_groups = (p.M + SHT_ROWS - 1) / SHT_ROWS;
        p.ksplit = k_blocks >= 2 ? 2u : 1u;
        for (uint32_t ks = SHT_MAX_KSPLIT; ks > 2; ks >>= 1)
            if (k_blocks >= 2 * ks && int(row_groups) <= shrink_tc_clusters(*dst, ks)) { p.ksplit = ks; break; }
        p.release_dependents = 1u;
        const uint32_t n_ctas = p.ksplit * ((rows + SHT_ROWS - 1) / SHT_ROWS);
        p.profile = (g_profile_buf && size_t(n_ctas) * 16 <= g_profile_words) ? g_profile_buf : nullptr;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(n_ctas);
        cfg.blockDim = dim3(SHT_THREADS);
        cfg.dynamicSmemBytes = SHT_SMEM_BYTES;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = p.ksplit;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cuda_status(cudaLaunchKernelEx(&cfg, lora_shrink_tc_kernel, map_x, map_a, p));
    }
    if (p.m_begin || p.m_count || p.n_tile_dest > 1) return ATLAS_B200_ERR_DIMS;      // a row range / several destinations: that kernel only
    if (mma_ok) {
        const uint32_t chunk = p.chunk ? p.chunk : uint32_t(SHM_CHUNK);
        const MmaShrinkGrid rule = mma_shrink_grid(n_slots, (p.max_rank + SHM_RANKS - 1) / SHM_RANKS, (p.M + chunk - 1) / chunk, std::min(p.M, chunk),
                                                   uint32_t(rt_sm_count()), beside);
        const uint32_t ksplit = p.ksplit = rule.ksplit;
        p.row_parts_log2 = rule.row_parts_log2;
        p.prefetch_ctas = rule.prefetch_ctas;
        dim3 grid(n_slots * ksplit, (p.max_rank + SHM_RANKS - 1) / SHM_RANKS, ((p.M + chunk - 1) / chunk) << p.row_parts_log2);
        if (grid.y > 65535 || grid.z > 65535) return ATLAS_B200_ERR_LIMIT;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(SHM_THREADS);
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;      // SHM_KSPLIT CTAs along x share one (slot, ranks, chunk)
        attr[0].val.clusterDim.x = ksplit;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cuda_status(cudaLaunchKernelEx(&cfg, lora_shrink_mma_kernel, p));
    }
    dim3 grid(n_slots, (p.max_rank + SHRINK_RT - 1) / SHRINK_RT, (p.M + SHRINK_TC - 1) / SHRINK_TC);
    if (grid.y > 65535 || grid.z > 65535) return ATLAS_B200_ERR_LIMIT;
    lora_shrink_grouped_kernel<<<grid, SHRINK_THREADS, 0, st>>>(p);
    return launch_status();
}

static int launch_expand(const ExpandParams& p, cudaStream_t st) {
    if (p.M == 0 || p.n_out == 0) return ATLAS_B200_OK;
    if (p.max_rank > EXPAND_MAX_RANK) return ATLAS_B200_ERR_LIMIT;
    if (p.max_rank % 8 == 0 && p.max_rank <= uint32_t(EXM_MAX_RANK) && aligned(p.xa, 8)) {
        // tensor cores (kernel_expand_mma.cuh) wherever xa rows can be read four ranks at a time and B_s fits in registers
        const uint32_t chunk = EXM_ROWS, chunks = (p.M + chunk - 1) / chunk, cols = (p.n_out + EXM_OUTS - 1) / EXM_OUTS;
        // CTAs sharing a chunk's runs: at most as many as it can have runs (one per slot that occurs, one more per sixteen
        // rows), and no more than eight CTAs per SM in all
        const uint32_t rows = std::min(p.M, chunk), most = (p.seq_slot ? std::min(rows, p.max_loras) : 0u) + (rows + 15) / 16;
        uint32_t splits = 1;
        while (splits * 2 <= most && uint64_t(cols) * chunks * splits * 2 <= uint64_t(rt_sm_count()) * 8) splits *= 2;
        const dim3 grid(cols, chunks * splits);
        if (grid.y > 65535) return ATLAS_B200_ERR_LIMIT;
        // One granule: six CTAs on an SM, with two registers too few, where five of them would not be resident at once.  Five / six (us):
        // dense base and 1000 tokens of 128 adapters of rank 16 x 14336 x 4096 (896 CTAs) 302 / 293; 256 tokens of 4 x 4096 x 4096 (512)
        // 30.7 / 32.1.
        if (p.max_rank <= 16)
            return uint64_t(grid.x) * grid.y > uint64_t(rt_sm_count()) * 5 ? launch_chained(lora_expand_mma_kernel<1, 6>, grid, EXM_THREADS, st, p, chunk, splits)
                                                                           : launch_chained(lora_expand_mma_kernel<1>, grid, EXM_THREADS, st, p, chunk, splits);
        if (p.max_rank <= 32) return launch_chained(lora_expand_mma_kernel<2>, grid, EXM_THREADS, st, p, chunk, splits);
        if (p.max_rank <= 64) return launch_chained(lora_expand_mma_kernel<4>, grid, EXM_THREADS, st, p, chunk, splits);
        return launch_chained(lora_expand_mma_kernel<8>, grid, EXM_THREADS, st, p, chunk, splits);
    }
    // rows per CTA: 32 for large batches (a CTA re-uses its B rows out of L1 while neighbouring rows share an adapter),
    // fewer while the grid would otherwise leave SMs without a CTA (a decode batch)
    ExpandParams q = p;
    const uint32_t col_blocks = (p.n_out + EXPAND_OUTS - 1) / EXPAND_OUTS;
    uint32_t rpc = EXPAND_ROWS;
    while (rpc > 1 && col_blocks * ((p.M + rpc - 1) / rpc) < 2u * uint32_t(rt_sm_count())) rpc >>= 1;
    q.rows_per_cta = rpc;
    dim3 grid(col_blocks, (p.M + rpc - 1) / rpc);
    if (grid.y > 65535) return ATLAS_B200_ERR_LIMIT;
    lora_expand_fold_kernel<<<grid, EXPAND_OUTS, 0, st>>>(q);
    return launch_status();
}

int apply_lora_bgmv(const void* x, const int32_t* seq_slot, const uint64_t* a_table, const uint64_t* b_table,
                    const float* scale_table, void* base_out, void* lora_xa, uint32_t n, uint32_t k_in,
                    uint32_t n_out, uint32_t max_rank, uint32_t x_row_stride, uint32_t out_row_stride,
                    uint32_t max_loras, cudaStream_t st) {
    if (n == 0) return ATLAS_B200_OK;
    if (!x || !seq_slot || !a_table || !b_table || !scale_table || !base_out || !lora_xa) return ATLAS_B200_ERR_NULL;
    if (k_in == 0 || n_out == 0 || max_rank == 0 || max_loras == 0) return ATLAS_B200_ERR_DIMS;
    if (x_row_stride < k_in || out_row_stride < n_out) return ATLAS_B200_ERR_DIMS;
    if (max_loras > 65535 || max_rank > EXPAND_MAX_RANK) return ATLAS_B200_ERR_LIMIT;
    if (!aligned(x, 2) || !aligned(base_out, 2) || !aligned(lora_xa, 2)) return ATLAS_B200_ERR_ALIGN;

    ShrinkParams sp{};
    sp.x = static_cast<const uint16_t*>(x);
    sp.seq_slot = seq_slot;
    sp.a_table = a_table;
    sp.b_table = nullptr;            // the reference's shrink looks at the A entry only (lora_bgmv.cu:63-65)
    sp.out = static_cast<uint16_t*>(lora_xa);
    sp.M = n; sp.k_in = k_in; sp.max_rank = max_rank; sp.x_row_stride = x_row_stride; sp.max_loras = max_loras;
    sp.post = 0.0f;
    int rc = launch_shrink(sp, max_loras, st);
    if (rc) return rc;

    ExpandParams ep{};
    ep.xa = static_cast<const uint16_t*>(lora_xa);
    ep.seq_slot = seq_slot;
    ep.a_table = a_table;            // a row whose shrink was skipped has no valid xa: skip its expand too
    ep.b_table = b_table;
    ep.scale_table = scale_table;
    ep.out = static_cast<uint16_t*>(base_out);
    ep.M = n; ep.n_out = n_out; ep.max_rank = max_rank; ep.out_row_stride = out_row_stride; ep.max_loras = max_loras;
    return launch_expand(ep, st);
}

int apply_lora_delta(const void* x, const void* a, const void* b, float scale, void* base_out, void* lora_xa,
                     void* lora_delta, uint32_t m, uint32_t k_in, uint32_t n_out, uint32_t max_rank, cudaStream_t st) {
    if (m == 0) return ATLAS_B200_OK;
    if (!x || !a || !b || !base_out || !lora_xa) return ATLAS_B200_ERR_NULL;
    if (k_in == 0 || n_out == 0 || max_rank == 0) return ATLAS_B200_ERR_DIMS;
    if (max_rank > EXPAND_MAX_RANK) return ATLAS_B200_ERR_LIMIT;

    ShrinkParams sp{};
    sp.x = static_cast<const uint16_t*>(x);
    sp.a_uniform = static_cast<const uint16_t*>(a);
    sp.out = static_cast<uint16_t*>(lora_xa);
    sp.M = m; sp.k_in = k_in; sp.max_rank = max_rank; sp.x_row_stride = k_in; sp.max_loras = 1;
    int rc = launch_shrink(sp, 1, st);
    if (rc) return rc;

    ExpandParams ep{};
    ep.xa = static_cast<const uint16_t*>(lora_xa);
    ep.b_uniform = static_cast<const uint16_t*>(b);
    ep.scale_uniform = scale;
    ep.out = static_cast<uint16_t*>(base_out);
    ep.delta_out = static_cast<uint16_t*>(lora_delta);
    ep.M = m; ep.n_out = n_out; ep.max_rank = max_rank; ep.out_row_stride = n_out; ep.max_loras = 1;
    return launch_expand(ep, st);
}

static int launch_simt_linear(const atlas_b200_linear_desc& d, cudaStream_t st) {
    SimtLinearParams p{};
    p.x = static_cast<const uint16_t*>(d.x);
    p.w_packed = static_cast<const uint8_t*>(d.w_packed);
    p.w_scale = static_cast<const uint8_t*>(d.w_scale);
    p.w_bf16 = static_cast<const uint16_t*>(d.w_bf16);
    p.y = static_cast<uint16_t*>(d.y);
    p.M = d.m; p.N = d.n; p.K = d.k; p.x_row_stride = d.x_row_stride; p.out_row_stride = d.out_row_stride;
    p.scale2 = d.w_bf16 ? 1.0f : d.scale2;
    dim3 grid((d.n + SIMT_TF - 1) / SIMT_TF, (d.m + SIMT_TM - 1) / SIMT_TM);
    if (grid.y > 65535) return ATLAS_B200_ERR_LIMIT;
    linear_simt_kernel<<<grid, 256, 0, st>>>(p);
    return launch_status();
}

// Shapes the tcgen05 path takes.  Everything here is a property of host-visible arguments.
// `wide`: also those for which it is only the faster of two paths — K a multiple of 32 (of 256 otherwise: the row strides of
// codes AND scales are then the 16-byte multiples TMA wants; with K = 32 n only the codes are, and the expansion warps read
// the scales themselves) and ranks up to 128 (64 otherwise).  What exists on this path alone (FP4 activations, placement,
// a forced path, the shrink by itself) keeps the narrow rule.
constexpr uint32_t TC_NARROW_RANK = 64;
static bool tc_eligible(const atlas_b200_linear_desc& d, bool wide) {
    DeviceState* dst = device_state();
    if (!dst || !dst->sm100 || !g_encode) return false;
    if (d.w_bf16) return false;                                   // dense base: a kernel of its own
    if (d.k % tc::KRAW != 0 && (!wide || d.k % 32 != 0 || d.k < uint32_t(tc::KRAW))) return false;
    if (d.x_row_stride % 8 != 0) return false;
    if (!aligned(d.x, 16) || !aligned(d.w_packed, 16) || !aligned(d.w_scale, 16)) return false;
    if (d.seq_slot) {
        if (d.max_rank > (wide ? uint32_t(tc::MAX_RANK_TC) : TC_NARROW_RANK) || d.max_rank % 8 != 0) return false;
        if (d.max_loras > tc::MAX_LORAS_TC) return false;
        if (!aligned(d.lora_t, 16)) return false;
    }
    if (!(d.scale2 != 0.0f) || !std::isfinite(d.scale2)) return false;
    return true;
}

// Bytes of `ws` the FP4-activation mode needs: packed codes [m, k/2] then scale bytes [m, k/16],
// the second at a 256-byte boundary.
static size_t act_fp4_codes_bytes(const atlas_b200_linear_desc& d) { return (size_t(d.m) * (d.k / 2) + 255) / 256 * 256; }
static size_t act_fp4_ws_bytes(const atlas_b200_linear_desc& d) { return act_fp4_codes_bytes(d) + size_t(d.m) * (d.k / 16); }

// The B side of the adapter pool can be described as one 3-D tensor [max_loras][n][max_rank]
static bool b_pool_is_strided(const atlas_b200_linear_desc& d) {
    return d.seq_slot && d.b_pool_base && d.b_slot_stride && d.b_slot_stride % 16 == 0 && aligned(d.b_pool_base, 16) &&
           d.max_rank % 8 == 0;
}

// Granules of B_s that one copy may bring: a copy of 128 rows takes as long for one of 16 ranks as for four of a slot.  With it, and one copy
// of masked t for a K block (us, by granules / so): 64 tokens of 64 adapters of rank 64 x 14336 x 4096 82.9 / 75.4 on the one-tile kernel.
static uint32_t granules_per_copy(const atlas_b200_linear_desc& d) {
    return !b_pool_is_strided(d) ? 1u : (d.max_rank % 64 == 0 ? 4u : (d.max_rank % 32 == 0 ? 2u : 1u));
}

// Where the shrink's masked-t tiles live in `ws` (tiles == nullptr: the fused kernel builds them itself from lora_t)
struct TTiles {
    uint16_t* tiles = nullptr;
    uint32_t cap = 0;          // blocks reserved per token tile (per half of one, for CTA pairs)
    uint32_t part_rows = 0;    // rows of a block: the token tile, or half of it for CTA pairs
};

// The tensor maps of a tcgen05 launch (`b`: one granule of B_s, `bw`: `lora_wide` of them).  `xrows` = token rows of an activation tile one CTA stages, `mt` = token
// tile, `l_gran_t` = bytes of one masked-t block as the shrink writes it ([part_rows x 16] BF16).
struct TcMaps { CUtensorMap x, w, s, b, bw, xs, t; };

// `t_blocks` = masked-t blocks per copy, `a4_scale_row` = scale bytes per row of a stage (FP4 activations).
static int encode_tc_maps(const atlas_b200_linear_desc& d, bool a4, uint32_t xrows, uint32_t mt, uint32_t l_gran_t,
                          const TTiles& tt, TcMaps& m, uint32_t t_blocks, uint32_t a4_scale_row = tc::KRAW / 16, uint32_t lora_wide = 1) {
    const CUtensorMapSwizzle scale_swizzle = a4_scale_row == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
    if (a4) {
        // the quantised activations in `ws`, in the weights' own layout
        const uint8_t* codes = static_cast<const uint8_t*>(d.ws);
        if (!encode_2d(&m.x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, d.k / 2, d.m, d.k / 2, tc::KRAW / 2, xrows,
                       CU_TENSOR_MAP_SWIZZLE_128B))
            return ATLAS_B200_ERR_DIMS;
        if (!encode_2d(&m.xs, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes + act_fp4_codes_bytes(d), d.k / 16, d.m, d.k / 16,
                       a4_scale_row, mt, scale_swizzle))
            return ATLAS_B200_ERR_DIMS;
    } else if (!encode_2d(&m.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d.x, d.k, d.m, uint64_t(d.x_row_stride) * 2, tc::KB, xrows,
                          CU_TENSOR_MAP_SWIZZLE_128B))
        return ATLAS_B200_ERR_DIMS;
    if (!encode_2d(&m.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, d.w_packed, d.k / 2, d.n, d.k / 2, tc::KRAW / 2, tc::FT,
                   CU_TENSOR_MAP_SWIZZLE_128B))
        return ATLAS_B200_ERR_DIMS;
    if (d.k % tc::KRAW != 0) m.s = m.w;      // scale rows of K/16 bytes: read by the expansion warps (Params::w_scale_rows)
    else if (!encode_2d(&m.s, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, d.w_scale, d.k / 16, d.n, d.k / 16, a4 ? a4_scale_row : tc::KRAW / 16, tc::FT,
                        a4 ? scale_swizzle : CU_TENSOR_MAP_SWIZZLE_NONE))
        return ATLAS_B200_ERR_DIMS;

    // B side of the adapter pool as one 3-D tensor [max_loras][n][max_rank]: box = some granules of one slot
    if (b_pool_is_strided(d)) {
        const uint64_t dims[3] = {d.max_rank, d.n, d.max_loras};
        const uint64_t strides[2] = {uint64_t(d.max_rank) * 2, uint64_t(d.b_slot_stride)};
        auto encode_b = [&](CUtensorMap& map, uint32_t granules) {
            const uint32_t box[3] = {16 * granules, tc::FT, 1};
            return encode_tiled(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d.b_pool_base, dims, strides, box,
                                granules == 4 ? CU_TENSOR_MAP_SWIZZLE_128B : (granules == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B));
        };
        if (!encode_b(m.bw, lora_wide)) return ATLAS_B200_ERR_DIMS;
        m.b = m.bw;
        if (lora_wide > 1 && !encode_b(m.b, 1)) return ATLAS_B200_ERR_DIMS;
    } else {
        m.b = m.bw = m.s;   // never dereferenced
    }
    if (!a4) m.xs = m.s;   // never dereferenced
    if (tt.tiles) {
        // the masked-t blocks are shared-memory images already: plain bytes, 256 to a row, `t_blocks` blocks per copy
        const uint64_t rows = uint64_t((d.m + mt - 1) / mt) * tt.cap * mt * 32 / 256;
        if (l_gran_t % 256 != 0 ||
            !encode_2d(&m.t, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, tt.tiles, 256, rows, 256, 256, t_blocks * l_gran_t / 256, CU_TENSOR_MAP_SWIZZLE_NONE))
            return ATLAS_B200_ERR_DIMS;
    } else {
        m.t = m.s;         // never dereferenced
    }
    return ATLAS_B200_OK;
}

// The shapes of the wide rule alone: their LoRA term was added row by row before they came to the fused kernels (isolate.cuh).
static bool isolates(const atlas_b200_linear_desc& d) {
    return d.seq_slot && (d.k % tc::KRAW != 0 || d.max_rank > TC_NARROW_RANK);
}

// What the shrink multiplies A_s x by, beside scale_s: t is in the unit of the MMA accumulator (no 2^8 with FP4 activations)
static float lora_post(const atlas_b200_linear_desc& d, bool act_fp4) { return act_fp4 ? 1.0f / d.scale2 : 1.0f / (d.scale2 * kWeightPreScale); }

// the launch constants both tcgen05 kernels share
static int fill_tc_params(const atlas_b200_linear_desc& d, bool a4, bool b_strided, const TTiles& tt, tc::Params& p) {
    p.b_pool_strided = b_strided ? 1u : 0u;
    p.b_pool_base = reinterpret_cast<unsigned long long>(d.b_pool_base);
    p.b_slot_stride = d.b_slot_stride;
    p.t_tile_cap = tt.tiles ? tt.cap : 0u;
    p.seq_slot = d.seq_slot;
    p.a_table = d.a_table;
    p.b_table = d.b_table;
    p.rank_table = d.rank_table;
    p.t = static_cast<const uint16_t*>(d.lora_t);
    p.y = static_cast<uint16_t*>(d.y);
    p.n_dest = d.n_dest ? d.n_dest : 1u;
    p.y_col0 = d.n_dest ? d.y_col_offset : 0u;
    bool rows_16b = d.out_row_stride % 8 == 0 && p.y_col0 % 8 == 0;
    for (uint32_t r = 0; r < p.n_dest; ++r) {
        p.y_dest[r] = static_cast<uint16_t*>(d.n_dest ? d.y_dest[r] : d.y);
        rows_16b = rows_16b && aligned(p.y_dest[r], 16);
    }
    if (d.n_dest && !rows_16b) return ATLAS_B200_ERR_ALIGN;
    p.staged_epilogue = rows_16b ? 1u : 0u;
    p.M = d.m; p.N = d.n; p.K = d.k; p.out_row_stride = d.out_row_stride;
    p.max_loras = d.max_loras; p.max_rank = d.max_rank;
    p.out_scale = a4 ? d.scale2 : d.scale2 * kWeightPreScale;
    p.w_scale_rows = d.k % tc::KRAW != 0 ? static_cast<const uint8_t*>(d.w_scale) : nullptr;
    p.k_split = 1;
    p.isolate = isolates(d) ? 1u : 0u;
    p.x = static_cast<const uint16_t*>(d.x);
    p.w_packed = static_cast<const uint8_t*>(d.w_packed);
    p.w_scale = static_cast<const uint8_t*>(d.w_scale);
    p.scale_table = d.scale_table;
    p.x_row_stride = d.x_row_stride;
    p.post = lora_post(d, a4);
    return ATLAS_B200_OK;
}

// How many clusters of (PAIR ? 2 : 1) x 1 x k_split CTAs of one kernel instance can be resident at once.  Clusters live
// inside one GPC, so fewer fit than the SM count suggests.  An occupancy query, answered by the runtime without touching
// the device; asked once per shape.  -1: the query failed.
template <int MT, bool A4, bool PAIR>
static int tc_active_clusters(int slot_idx, uint32_t k_split) {
    using C = tc::Cfg<MT, A4, PAIR>;
    DeviceState* dst = device_state();
    if (!dst) return -1;
    slot_idx += (A4 ? 5 : 0) + (PAIR ? 10 : 0);
    int (&known)[20][9] = dst->known_clusters;
    if (k_split > 8) return -1;
    if (known[slot_idx][k_split] == 0) {
        if (!dst->tc_attr_set[slot_idx]) {
            if (cudaFuncSetAttribute(tc::nvfp4_lora_linear_tc_kernel<MT, A4, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     C::SMEM_BYTES) != cudaSuccess) {
                (void)cudaGetLastError();
                return -1;
            }
            dst->tc_attr_set[slot_idx] = true;
        }
        cudaLaunchConfig_t q{};
        q.gridDim = dim3(PAIR ? 2 : 1, 1, k_split);
        q.blockDim = dim3(tc::NUM_THREADS);
        q.dynamicSmemBytes = C::SMEM_BYTES;
        cudaLaunchAttribute qa[1];
        qa[0].id = cudaLaunchAttributeClusterDimension;
        qa[0].val.clusterDim.x = PAIR ? 2 : 1;
        qa[0].val.clusterDim.y = 1;
        qa[0].val.clusterDim.z = k_split;
        q.attrs = qa;
        q.numAttrs = 1;
        int n = 0;
        known[slot_idx][k_split] =
            cudaOccupancyMaxActiveClusters(&n, tc::nvfp4_lora_linear_tc_kernel<MT, A4, PAIR>, &q) == cudaSuccess && n > 0 ? n : -1;
        (void)cudaGetLastError();
    }
    return known[slot_idx][k_split];
}

static int tc_active_clusters_of(uint32_t mt, bool a4, bool pair, uint32_t k_split) {
#define ATLAS_OCC(MT_, I_) \
    if (mt == MT_) return a4 ? (pair ? tc_active_clusters<MT_, true, (MT_ >= 128)>(I_, k_split) : tc_active_clusters<MT_, true, false>(I_, k_split)) \
                             : (pair ? tc_active_clusters<MT_, false, (MT_ >= 128)>(I_, k_split) : tc_active_clusters<MT_, false, false>(I_, k_split));
    ATLAS_OCC(16, 0) ATLAS_OCC(32, 1) ATLAS_OCC(64, 2) ATLAS_OCC(128, 3) ATLAS_OCC(256, 4)
#undef ATLAS_OCC
    return -1;
}

template <int MT, bool A4, bool PAIR, bool SROWS, bool ISO>
static int launch_tc_as(const atlas_b200_linear_desc& d, int slot_idx, const ShrinkParams* shrink, const TTiles& tt,
                     uint32_t k_split, cudaStream_t st) {
    const bool after_shrink = shrink != nullptr;     // the shrink is launched from here, once the launch shape is final
    using C = tc::Cfg<MT, A4, PAIR>;
    DeviceState* dst = device_state();
    if (!dst) return ATLAS_B200_ERR_ARCH;
    slot_idx += (A4 ? 5 : 0) + (PAIR ? 10 : 0) + (SROWS ? 20 : (ISO ? 40 : 0));
    if (!dst->tc_attr_set[slot_idx]) {
        cudaError_t e = cudaFuncSetAttribute(tc::nvfp4_lora_linear_tc_kernel<MT, A4, PAIR, SROWS, ISO>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (e != cudaSuccess) return cuda_status(e);
        dst->tc_attr_set[slot_idx] = true;
    }
    TcMaps maps;
    const bool b_strided = b_pool_is_strided(d);
    const uint32_t lora_wide = granules_per_copy(d);
    {
        const int rc = encode_tc_maps(d, A4, C::XROWS, MT, C::L_GRAN_T, tt, maps, 4, tc::KRAW / 16, lora_wide);
        if (rc) return rc;
    }
    const CUtensorMap &map_x = maps.x, &map_w = maps.w, &map_s = maps.s, &map_b = maps.b, &map_bw = maps.bw, &map_xs = maps.xs, &map_t = maps.t;

    tc::Params p{};
    {
        const int rc = fill_tc_params(d, A4, b_strided, tt, p);
        if (rc) return rc;
    }
    p.lora_wide = lora_wide;
    dim3 grid((d.n + tc::FT - 1) / tc::FT, (d.m + MT - 1) / MT);
    if (PAIR) grid.x = (grid.x + 1u) & ~1u;      // whole pairs: a CTA past the last feature loads zeros and stores nothing
    // split K: k_split CTAs along z form a cluster (times two for pairs), share one tile and exchange partial sums
    // (the staging area holds those of every split up to this one)
    if (k_split > uint32_t(C::MAX_SPLIT)) return ATLAS_B200_ERR_LIMIT;
    grid.z = k_split;
    p.k_split = k_split;
    t_last_shape[0] = MT; t_last_shape[1] = PAIR ? 1u : 0u; t_last_shape[2] = k_split; t_last_shape[3] = tt.tiles ? 1u : 0u;
    t_last_shape[4] = 0u; t_last_shape[5] = 0u; t_last_shape[6] = 0u; t_last_shape[7] = 0u;
    if (shrink) {
        // Gaps while the shrink runs, for pairs whose CTAs contract more than it takes (their MMAs leave no idle cycles).  Two or three CTAs
        // to a long K, up to 64 granules: before every stage, up to rank 16 before every other.  Without / before every other / before every
        // stage / before every stage of the whole loop (us): 512 tokens x 4096 x 14336 8 of rank 16 59.3 / 52.3 / 53.4 / 57.9, 16 of rank
        // 32 in sequences 87.5 / 74.4 / 73.2 / 79.2, 280 tokens 8 of rank 32 in sequences 70.4 / 61.7 / 58.7 / 59.7, 400 x 2560 x 6912 8 of
        // rank 16 31.1 / 27.8 / 28.4 / 29.5; but 64 of rank 64 (several rounds of the shrink) 512 x 4096 x 14336 157.8 /
        // 159.2, four CTAs (130 x 4096 x 14336) 34.7 / 36.5, 2048 of K to one of two (512 x 4096 x 4096) 25.2 / 25.8, and single CTAs,
        // which wait for shared memory (700 x 3072 x 9216) 38.7 / 41.6.
        // One CTA: before every fourth, and only for more tokens than a tile, whose shrink is the longer one, of few granules.  Without /
        // so / before every other stage: 1000 x 4096 x 14336 8 of rank 32 in sequences 125.5 / 114.8 / 112.7, of rank 16 95.2 / 90.7 / 90.9,
        // 512 x 8192 x 6144 8 of rank 32 in sequences 52.1 / 47.5 / 47.1, of rank 16 (the dearest, a per cent) 42.9 / 43.3 / 43.5; but 256
        // x 17408 x 5120 16 of rank 32 42.5 / 42.6 / 43.1, one of rank 16 (1000 x 4096 x 6144) 42.6 / 43.4 / 43.5, 32 of rank 32 (512 x
        // 8192 x 8192) 72.6 / 73.4 / 73.7, K = 4096 (1000 x 4096, 16 of rank 32) 45.7 / - / 46.1.
        const uint64_t granules = uint64_t(d.max_loras) * ((d.max_rank + 15) / 16);
        p.leave_gaps = 0u;
        if (PAIR && MT >= 256 && !A4 && d.k > 4096 && d.m <= 1024) {
            if (k_split == 1) p.leave_gaps = d.m > uint32_t(MT) && granules > 1 && granules <= 32 ? 4u : 0u;
            else p.leave_gaps = k_split <= 3 && d.k > 2048 * k_split && granules <= 64 ? (d.max_rank > 16 ? 1u : 2u) : 0u;
        }
        t_last_shape[6] = p.leave_gaps ? 1u : 0u;
        // A small batch: the mma.sync shrink releases this kernel as soon as it is resident, which then runs beside it.  A large one:
        // the tcgen05 shrink fills its SMs and releases this kernel at the same point, whose CTAs then take SMs that are free or
        // become so; the mma.sync shrink, where it has to stand in, keeps the machine to itself.
        const uint32_t main_ctas = grid.x * grid.y * grid.z;
        const int rc = launch_shrink(*shrink, d.max_loras, st, d.m > 1024 ? MachineBeside::none
                                     : (main_ctas * 3 <= uint32_t(rt_sm_count()) * 2 ? MachineBeside::part : MachineBeside::tiles));
        if (rc) return rc;
    }
    p.profile = (g_profile_buf && size_t(grid.x) * grid.y * tc::PROFILE_WORDS <= g_profile_words) ? g_profile_buf : nullptr;
    if (grid.y > 65535) return ATLAS_B200_ERR_LIMIT;
    // Launched as a programmatic dependent of the shrink that precedes it in the stream: its CTAs
    // may start while the shrink still runs (see above) and wait for the shrink's completion only
    // where they first read t, after the base K loop.
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(tc::NUM_THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n_attr = 0;
    if (PAIR || k_split > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = PAIR ? 2 : 1;
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr].val.clusterDim.z = k_split;
        ++n_attr;
    }
    p.chained = d.seq_slot ? 0u : 1u;
    if (after_shrink || p.chained) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    p.wait_for_shrink = after_shrink ? 1u : 0u;
    return cuda_status(cudaLaunchKernelEx(&cfg, tc::nvfp4_lora_linear_tc_kernel<MT, A4, PAIR, SROWS, ISO>, map_x, map_w, map_s, map_b, map_bw, map_xs, map_t, p));
}

template <int MT, bool A4, bool PAIR>
static int launch_tc(const atlas_b200_linear_desc& d, int slot_idx, const ShrinkParams* shrink, const TTiles& tt,
                     uint32_t k_split, cudaStream_t st) {
    if constexpr (!A4)
    {
        if (d.k % tc::KRAW != 0) return launch_tc_as<MT, false, PAIR, true, true>(d, slot_idx, shrink, tt, k_split, st);
        if (isolates(d)) return launch_tc_as<MT, false, PAIR, false, true>(d, slot_idx, shrink, tt, k_split, st);
    }
    return launch_tc_as<MT, A4, PAIR, false, false>(d, slot_idx, shrink, tt, k_split, st);
}

// ---- the persistent form (kernel_tc_persist.cuh): one cluster of two CTAs per pair of SMs, a static tile loop ----
// instance index: 0 = <256, 1, A16>, 1 = <256, 1, A4>, 2 = <192, 2, A16>, 3 and 4 = 0 and 2 for calls that isolate
template <int MT, int G, bool A4, bool ISO = false>
static int persist_resident_clusters(int idx) {
    using C = tc::PCfg<MT, G, A4>;
    DeviceState* dst = device_state();
    if (!dst) return -1;
    if (dst->persist_clusters[idx] == 0) {
        if (!dst->persist_attr_set[idx]) {
            if (cudaFuncSetAttribute(tc::nvfp4_lora_linear_tc_persistent_kernel<MT, G, A4, ISO>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) {
                (void)cudaGetLastError();
                return -1;
            }
            dst->persist_attr_set[idx] = true;
        }
        cudaLaunchConfig_t q{};
        q.gridDim = dim3(2, 1, 1);
        q.blockDim = dim3(tc::P_NUM_THREADS);
        q.dynamicSmemBytes = C::SMEM_BYTES;
        cudaLaunchAttribute qa[1];
        qa[0].id = cudaLaunchAttributeClusterDimension;
        qa[0].val.clusterDim.x = 2;
        qa[0].val.clusterDim.y = 1;
        qa[0].val.clusterDim.z = 1;
        q.attrs = qa;
        q.numAttrs = 1;
        int n = 0;
        dst->persist_clusters[idx] =
            cudaOccupancyMaxActiveClusters(&n, tc::nvfp4_lora_linear_tc_persistent_kernel<MT, G, A4, ISO>, &q) == cudaSuccess && n > 0 ? n : -1;
        (void)cudaGetLastError();
    }
    return dst->persist_clusters[idx];
}

// tiles of one launch: pairs of feature tiles x token passes
template <int MT, int G>
static uint32_t persist_tiles(const atlas_b200_linear_desc& d) {
    const uint32_t n_fpairs = ((d.n + tc::FT - 1) / tc::FT + 1) / 2;
    const uint32_t n_passes = (d.m + MT * G - 1) / (MT * G);
    return n_fpairs * n_passes;
}

template <int MT, int G, bool A4, bool ISO = false>
static int launch_tc_persist(const atlas_b200_linear_desc& d, int idx, const ShrinkParams* shrink, const TTiles& tt, cudaStream_t st) {
    using C = tc::PCfg<MT, G, A4>;
    const int clusters = persist_resident_clusters<MT, G, A4, ISO>(idx);
    if (clusters <= 0) return ATLAS_B200_ERR_DIMS;
    const uint32_t lora_wide = std::min(granules_per_copy(d), uint32_t(C::LB));
    TcMaps maps;
    {
        const int rc = encode_tc_maps(d, A4, C::XROWS, MT, C::L_GRAN_T, tt, maps, C::LB, tc::A4_SCALE_ROW, lora_wide);
        if (rc) return rc;
    }
    tc::Params p{};
    {
        const int rc = fill_tc_params(d, A4, b_pool_is_strided(d), tt, p);
        if (rc) return rc;
    }
    if (!p.staged_epilogue) return ATLAS_B200_ERR_ALIGN;
    tc::PParams pp{};
    pp.n_fpairs = ((d.n + tc::FT - 1) / tc::FT + 1) / 2;
    pp.n_passes = (d.m + MT * G - 1) / (MT * G);
    pp.n_tiles = pp.n_fpairs * pp.n_passes;
    p.lora_wide = lora_wide;
    const uint32_t pairs = std::min<uint32_t>(uint32_t(clusters), pp.n_tiles);
    t_last_shape[0] = MT; t_last_shape[1] = 1u; t_last_shape[2] = 1u; t_last_shape[3] = tt.tiles ? 1u : 0u;
    t_last_shape[4] = uint32_t(G); t_last_shape[5] = pairs; t_last_shape[6] = 0u; t_last_shape[7] = 0u;
    if (shrink) {
        const int rc = launch_shrink(*shrink, d.max_loras, st, d.m > 1024 ? MachineBeside::none : MachineBeside::all);
        if (rc) return rc;
    }
    p.profile = (g_profile_buf && size_t(pairs) * 2 * tc::PROFILE_WORDS <= g_profile_words) ? g_profile_buf : nullptr;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pairs * 2, 1, 1);
    cfg.blockDim = dim3(tc::P_NUM_THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n_attr = 0;
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 2;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
    p.chained = d.seq_slot ? 0u : 1u;
    if (shrink || p.chained) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    p.wait_for_shrink = shrink ? 1u : 0u;
    return cuda_status(cudaLaunchKernelEx(&cfg, tc::nvfp4_lora_linear_tc_persistent_kernel<MT, G, A4, ISO>, maps.x, maps.w, maps.s, maps.b, maps.bw,
                                          maps.xs, maps.t, p, pp));
}

// ---- the smallest batches (kernel_decode_mma.cuh) ----
template <int TILES, int NT, int WARPS, bool BASE>
static int launch_decode_form(const atlas_b200_linear_desc& d, const ShrinkParams* shrink, bool tma, cudaStream_t st) {
    tc::Params p{};
    int rc = fill_tc_params(d, false, false, TTiles{}, p);
    if (rc) return rc;
    DecodeParams w{};
    w.x = static_cast<const uint16_t*>(d.x);
    w.w_packed = static_cast<const uint8_t*>(d.w_packed);
    w.w_scale = static_cast<const uint8_t*>(d.w_scale);
    w.x_row_stride = d.x_row_stride;
    const uint32_t ctas = (d.n + 16 * TILES - 1) / (16 * TILES);
    t_last_shape[0] = 8u; t_last_shape[1] = 0u; t_last_shape[2] = 1u; t_last_shape[3] = 0u; t_last_shape[4] = 0u; t_last_shape[5] = 0u; t_last_shape[6] = 0u;
    t_last_shape[7] = tma ? 1u : 0u;
    if (shrink) {
        rc = launch_shrink(*shrink, d.max_loras, st, ctas * 3 <= uint32_t(rt_sm_count()) * 2 ? MachineBeside::part : MachineBeside::all);
        if (rc) return rc;
    }
    p.wait_for_shrink = shrink ? 1u : 0u;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(32 * WARPS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = shrink || BASE ? 1 : 0;
    if constexpr (NT == 1)
        if (tma) {
            using R = DcmRing<TILES, WARPS>;
            const auto kernel = nvfp4_lora_decode_mma_kernel<TILES, 1, WARPS, true, BASE>;
            DeviceState* dst = device_state();
            if (!dst) return ATLAS_B200_ERR_ARCH;
            bool& set = dst->decode_attr_set[(TILES - 1) * 4 + (WARPS == 8 ? 2 : 0) + (BASE ? 1 : 0)];
            if (!set) {
                const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM_BYTES);
                if (e != cudaSuccess) return cuda_status(e);
                set = true;
            }
            CUtensorMap map_w, map_s;
            if (!encode_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, d.w_packed, d.k / 2, d.n, d.k / 2, 128, R::ROWS, CU_TENSOR_MAP_SWIZZLE_128B) ||
                !encode_2d(&map_s, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, d.w_scale, d.k / 16, d.n, d.k / 16, 8 * WARPS, R::ROWS,
                           WARPS == 8 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B))
                return ATLAS_B200_ERR_DIMS;
            cfg.blockDim = dim3(32 * (WARPS + 1));
            cfg.dynamicSmemBytes = R::SMEM_BYTES;
            return cuda_status(cudaLaunchKernelEx(&cfg, kernel, w, p, map_w, map_s));
        }
    CUtensorMap none;
    std::memset(&none, 0, sizeof(none));                      // never dereferenced
    return cuda_status(cudaLaunchKernelEx(&cfg, nvfp4_lora_decode_mma_kernel<TILES, NT, WARPS, false, BASE>, w, p, none, none));
}

// Weights by TMA (one n-tile; K of whole boxes): the warps' loads then are those of x, t and B alone, which is what the shrink beside this
// kernel and the granules behind it gain from; a small layer pays for the barriers and the longer way of its first bytes.  By the warps'
// loads / TMA (us), granules of the batch: 4096 x 4096 8 9.2 / 10.1, 12 10.0 / 10.8, 16 12.2 / 11.0, 32 16.2 / 12.9; 5120 x 5120 8 13.4 /
// 13.5, 16 14.8 / 14.2, 32 18.7 / 15.7; 14336 x 4096 8 17.8 / 18.3, 16 22.9 / 20.4, 32 28.5 / 23.7; 4096 x 14336 8 18.5 / 18.1, 16 26.1 /
// 18.6, 24 32.4 / 19.9; but 11008 x 4096 16 18.7 / 19.1, 2560 x 2560 16 8.2 / 9.0, 64 13.7 / 13.6.  Large layers whatever the batch: 8192 x
// 8192 one token, no adapters 15.7 / 15.3, 28672 x 8192 44.8 / 42.8, 8192 x 28672 48.1 / 43.3, 8 tokens of 8 x 64 x 28672 x 8192 73 / 59.
// What a batch uses of the granules that it could is not known on the host.  8 tokens of 32 x 32, all different / most without an adapter:
// 4096 x 4096 15.2 / 12.6, 10.0 / 10.8; 5120 x 5120 17.3 / 15.8, 13.9 / 13.6; 8192 x 4096 18.8 / 18.7, 13.3 / 13.7; 14336 x 4096 27.8 /
// 22.7, 19.1 / 19.4; 4096 x 14336 33.2 / 20.9, 25.7 / 19.1; 4 tokens of one among 32 x 128, 3072 x 14336 18.6 / 19.9.
static bool decode_by_tma(const atlas_b200_linear_desc& d) {
    const uint64_t weights = uint64_t(d.n) * d.k, granules = d.seq_slot ? std::min(d.max_loras, d.m) * ((d.max_rank + 15) / 16) : 0u;
    return d.k % tc::KRAW == 0 && (weights >= 1u << 26 || (weights >= 1u << 24 && granules >= 16));
}
template <int TILES, int NT, int WARPS>
static int launch_decode_as(const atlas_b200_linear_desc& d, const ShrinkParams* shrink, cudaStream_t st) {
    const bool tma = NT == 1 && decode_by_tma(d);
    if constexpr (NT == 1)
        if (!d.seq_slot) return launch_decode_form<TILES, NT, WARPS, true>(d, shrink, tma, st);
    return launch_decode_form<TILES, NT, WARPS, false>(d, shrink, tma, st);
}

// Where it is the faster one, both sides measured at cold L2 (us, this kernel / tcgen05):
//   no adapters          2 tokens    1024 x 4096 4.2/6.2   4096 x 4096 5.8/8.8    14336 x 4096 14.8/17.7  4096 x 14336 14.5/17.6  28672 x 8192 42/61
//                        16 tokens   1024 x 4096 5.9/6.6   4096 x 4096 8.2/9.0    14336 x 4096 19.3/17.8  4096 x 14336 22.9/18.1  28672 x 8192 60/61
//   8 of rank 16         2 tokens    1024 x 4096 6.1/9.4   4096 x 4096 7.6/12.1   14336 x 4096 17.3/21.1  4096 x 14336 16.1/20.7  28672 x 8192 47/65
//                        16 tokens   1024 x 4096 7.7/10.5  4096 x 4096 11.6/12.8  14336 x 4096 24.6/22.1  4096 x 14336 28.8/21.9  28672 x 8192 69/67
//   32 of rank 64        8 tokens    1024 x 4096 13.5/13.5 4096 x 4096 16.2/17.6  14336 x 4096 29.5/26.5  4096 x 14336 29.6/31.4  28672 x 8192 66/73
// With adapters the shrink runs beside it, and this kernel leaves that less of the memory system than the tcgen05 form does.
// Without adapters, and for N >= 2 K up to eight tokens and beyond them up to 32 granules, it is taken whatever the sizes, although the
// other is ahead at both tables' ends (16 tokens, no adapters, x 4096 x 14336; 8 of 32 x 64 x 14336 x 4096): a row without an adapter has
// the bits of the call without adapters, and a token's do not depend on the adapters that are loaded, only where all of these run here.
// N >= 2 K, beyond that: a granule (16 ranks of a slot) costs it some 0.3 us more than the other, against what it gains on the weights, most
// where those are more than one wave of tiles there.
// N < 2 K, up to eight tokens: it loses only to many granules and where a long K meets so few features that the other splits it (8 tokens
// of 32 of rank 16 x 4096 x 14336 24.3/21.7, 2 of rank 64 22.0/21.2; but of 32 of rank 64 29.6/31.4, 4 of rank 32 x 13824 x 14336 43/56).
// Beyond eight granules it is ahead or even there again, its weights coming by TMA from 2^24 of them on, the other's granules a chain of
// their own behind the loop: 8 tokens, 16 granules of rank 32 / 32 of rank 64, x 136 x 14336 14.4/17.2, 16.3/17.7, x 1024 x 14336 14.9/16.2,
// 19.1/18.7, x 2048 x 14336 16.5/17.8, 20.3/19.5, x 4096 x 14336 19.9/21.7, 22.8/22.6; 12 granules (6 tokens of 8 of rank 32), still by
// the warps' loads, x 136 x 14336 13.2/16.7, but x 3072 x 14336 20.8/18.7.
// Beyond eight tokens (two n-tiles, no weights by TMA) both are estimated, in us: this kernel by its weights, the length of a CTA's loop and
// its granules, the other by the K blocks a CTA takes one behind the other; measured from K = 1024 on.  12 tokens, 8 of rank 16 x 1024 x
// 4096 7.3/10.3, x 4096 x 4096 10.9/12.7, x 8192 x 8192 21.9/22.5, but x 5120 x 5120 15.0/14.1 and 32 of rank 64 x 4096 x 4096 20.6/18.7.
static bool decode_pays(const atlas_b200_linear_desc& d) {
    if (d.m > uint32_t(DCM_MAX_TOKENS)) return false;
    if (!d.seq_slot) return true;
    const uint32_t granules = std::min(d.m, d.max_loras) * ((d.max_rank + 15) / 16), tiles = (d.n + tc::FT - 1) / tc::FT, sms = uint32_t(rt_sm_count());
    if (uint64_t(d.n) >= 2ull * d.k) return d.m <= 8 || granules <= std::max(32u, d.k / (tiles > sms ? 80u : 128u));
    if (d.m <= 8) return granules < 64 && (uint64_t(d.m) * d.k <= (d.max_rank > 32 ? 86400u : 112000u) || d.n > 5120 || granules > 8);
    if (d.k < 1024) return false;
    const uint32_t split = std::max(1u, std::min(std::min(sms / tiles, 8u), d.k / uint32_t(tc::KRAW))), waves = (tiles * split + sms - 1) / sms;
    const float k = float(d.k) / 1024.0f, g = float(granules);
    const float here = 4.7f + 0.26f * k * float(d.n) / 1024.0f + 0.27f * k + g * (0.07f * std::max(float(d.n) / 4096.0f, 1.0f) + 0.017f * k);
    const float there = 8.1f + 3.4f * k * float(waves) / float(split) + 0.04f * g * float(waves);
    return here < 0.95f * there;                 // (a batch may use fewer adapters than it could, which the other gains on)
}

static int launch_decode(const atlas_b200_linear_desc& d, const ShrinkParams* shrink, cudaStream_t st) {
    // Sixteen warps fit on an SM.  Sixteen features per CTA instead of 32 where the two CTAs of eight warps that fit on an SM then still
    // cover them in one wave; and four warps to a CTA where even with 32 features they do not: four such CTAs on an SM are one wave up
    // to 18944 features, and beyond, CTAs at different points of their lives fill each other's gaps.  Eight / four warps, 1 and 8
    // tokens, 8 adapters of rank 16 (us): 11008 x 4096 15.9 / 14.0, 21.4 / 16.7; 14336 x 4096 17.9 / 16.3, 22.1 / 19.5; 28672 x 8192
    // 48.1 / 45.4, 56.8 / 52.3; but 8192 x 8192 (256 CTAs) 17.1 / 18.6, 19.7 / 25.9.
    // The batch's granules are shared by half as many warps then, which the longer loop pays for less and less as K grows.  Eight /
    // four warps (us) by granules: 14336 x 4096, 16 23.6 / 21.1, 32 28.7 / 27.9, 64 33.4 / 37.1; x 5120, 16 28.5 / 26.1, 32 33.4 / 34.2;
    // x 6912, 8 29.2 / 28.0, 16 32.9 / 36.8; x 2048, 32 20.8 / 18.8.  Beyond eight tokens, 8 and 16: 14336 x 4096 25.4 / 24.3, 28.2 /
    // 28.3, x 5120 29.4 / 29.0, 31.5 / 37.1, x 6912 36.0 / 39.0, 39.5 / 48.2, but 11008 x 4096, hardly more than a wave of eight-warp
    // CTAs, 25.1 / 20.7, 28.1 / 24.4.  Beyond one wave of four-warp CTAs, 8 and 16 whatever K: 28672 x 4096 34.5 / 34.0, 42.9 / 45.2, x
    // 8192 55.0 / 54.7, 60.9 / 64.1, 16 tokens 71.1 / 69.7, 78.9 / 89.5; 8 of one adapter x 4096 31.2 / 32.5.
    // (Both forms give the same bits.)
    const bool few = d.m <= 8;
    const uint32_t slots = 2u * uint32_t(rt_sm_count());
    const uint64_t granules = d.seq_slot ? std::min(d.max_loras, d.m) * ((d.max_rank + 15) / 16) : 0u, k = few ? std::max(d.k, 4096u) : d.k;
    const bool four = d.n > 64u * slots ? granules <= 8u && d.max_rank <= 64u
                                        : granules * k * k * k * (few ? 1u : (d.n <= 40u * slots ? 2u : 4u)) <= 32ull * 4096 * 4096 * 4096;
    if (d.n <= 16u * slots) return few ? launch_decode_as<1, 1, 8>(d, shrink, st) : launch_decode_as<1, 2, 8>(d, shrink, st);
    if (d.n <= 32u * slots || !four) return few ? launch_decode_as<2, 1, 8>(d, shrink, st) : launch_decode_as<2, 2, 8>(d, shrink, st);
    return few ? launch_decode_as<2, 1, 4>(d, shrink, st) : launch_decode_as<2, 2, 4>(d, shrink, st);
}

// ---- dense-BF16 base on the tensor cores (kernel_dense_tc.cuh) ----
// K: rows of 16-byte multiples, which is what TMA wants (it fills a last, partial K block with zeros); a forced tcgen05 path
// keeps to whole blocks
static bool dense_tc_eligible(const atlas_b200_linear_desc& d) {
    DeviceState* dst = device_state();
    const uint32_t k_unit = (d.flags & ATLAS_B200_FLAG_FORCE_TCGEN05) ? uint32_t(tc::KB) : 8u;
    return dst && dst->sm100 && g_encode && d.w_bf16 && d.k % k_unit == 0 && d.k >= uint32_t(tc::KB) && d.x_row_stride % 8 == 0 && aligned(d.x, 16) &&
           aligned(d.w_bf16, 16) && !d.n_dest;
}

template <int MT>
static int launch_dense_tc_mt(const atlas_b200_linear_desc& d, int idx, uint32_t k_split, bool after_shrink, cudaStream_t st) {
    using C = tc::DCfg<MT>;
    DeviceState* dst = device_state();
    if (!dst->dense_attr_set[idx]) {
        cudaError_t e = cudaFuncSetAttribute(tc::dense_bf16_linear_tc_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (e != cudaSuccess) return cuda_status(e);
        dst->dense_attr_set[idx] = true;
    }
    CUtensorMap map_x, map_w;
    if (!encode_2d(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d.x, d.k, d.m, uint64_t(d.x_row_stride) * 2, tc::KB, MT, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d.w_bf16, d.k, d.n, uint64_t(d.k) * 2, tc::KB, tc::FT, CU_TENSOR_MAP_SWIZZLE_128B))
        return ATLAS_B200_ERR_DIMS;
    tc::DParams p{};
    p.y = static_cast<uint16_t*>(d.y);
    p.M = d.m; p.N = d.n; p.K = d.k; p.out_row_stride = d.out_row_stride; p.k_split = k_split;
    p.after_shrink = after_shrink ? 1u : 0u;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((d.n + tc::FT - 1) / tc::FT, (d.m + MT - 1) / MT, k_split);
    if (cfg.gridDim.y > 65535) return ATLAS_B200_ERR_LIMIT;
    cfg.blockDim = dim3(tc::D_THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = k_split;
    cfg.attrs = attr;
    cfg.numAttrs = k_split > 1 ? 2 : 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, tc::dense_bf16_linear_tc_kernel<MT>, map_x, map_w, p));
}

static int launch_dense_tc(const atlas_b200_linear_desc& d, bool after_shrink, cudaStream_t st) {
    uint32_t mt = 16;
    while (mt < 128 && mt < d.m) mt <<= 1;
    // few output tiles (a decode batch): CTAs along z share a tile's K so that every SM streams weights
    const uint32_t tiles = ((d.n + tc::FT - 1) / tc::FT) * ((d.m + mt - 1) / mt);
    uint32_t k_split = std::max(1u, std::min(std::min(uint32_t(rt_sm_count()) / std::max(tiles, 1u), 8u), d.k / uint32_t(tc::KB)));
    while (k_split & (k_split - 1)) --k_split;           // a power of two: clusters of 1, 2, 4 or 8
    t_last_shape[0] = mt; t_last_shape[1] = 0u; t_last_shape[2] = k_split; t_last_shape[3] = 0u; t_last_shape[4] = 0u; t_last_shape[5] = 0u; t_last_shape[6] = 0u;
    t_last_shape[7] = 0u;
    if (mt == 16) return launch_dense_tc_mt<16>(d, 0, k_split, after_shrink, st);
    if (mt == 32) return launch_dense_tc_mt<32>(d, 1, k_split, after_shrink, st);
    if (mt == 64) return launch_dense_tc_mt<64>(d, 2, k_split, after_shrink, st);
    return launch_dense_tc_mt<128>(d, 3, k_split, after_shrink, st);
}

static int validate_linear(const atlas_b200_linear_desc& d) {
    if (!d.x || (!d.y && !d.n_dest)) return ATLAS_B200_ERR_NULL;
    if (d.n_dest > uint32_t(tc::MAX_DEST)) return ATLAS_B200_ERR_LIMIT;
    for (uint32_t r = 0; r < d.n_dest; ++r)
        if (!d.y_dest[r]) return ATLAS_B200_ERR_NULL;
    if (d.n_dest && uint64_t(d.y_col_offset) + d.n > d.out_row_stride) return ATLAS_B200_ERR_DIMS;
    if (!d.w_bf16 && (!d.w_packed || !d.w_scale)) return ATLAS_B200_ERR_NULL;
    if (d.k == 0 || d.n == 0) return ATLAS_B200_ERR_DIMS;
    if (!d.w_bf16 && d.k % 16 != 0) return ATLAS_B200_ERR_DIMS;   // NVFP4 scale groups are 16 wide
    if (d.x_row_stride < d.k || d.out_row_stride < d.n) return ATLAS_B200_ERR_DIMS;
    if (d.seq_slot) {
        if (!d.a_table || !d.b_table || !d.scale_table || !d.lora_t) return ATLAS_B200_ERR_NULL;
        if (d.max_loras == 0 || d.max_rank == 0) return ATLAS_B200_ERR_DIMS;
        if (d.max_loras > 65535 || d.max_rank > EXPAND_MAX_RANK) return ATLAS_B200_ERR_LIMIT;
    }
    if ((d.flags & ATLAS_B200_FLAG_FORCE_SIMT) && (d.flags & ATLAS_B200_FLAG_FORCE_TCGEN05)) return ATLAS_B200_ERR_DIMS;
    return ATLAS_B200_OK;
}

// A call that stops after the shrink: rows [row_begin, row_begin + row_count) of the batch, masked-t tiles written into
// n_dest scratch buffers laid out like d.ws (see atlas_b200_lora_shrink_tiles).
struct ShrinkOnly {
    uint32_t row_begin, row_count, n_dest;
    void* const* ws_dest;
};

// The launch shape of a call on the tensor-core path: a function of the descriptor's sizes and addresses and of `flags`
// (d.flags, or those of another call that shares its scratch).
struct TcPlan {
    bool decode = false;           // kernel_decode_mma.cuh; of the rest only `tt` (none) is meant
    uint32_t mt = 16, k_split = 1; // token tile; CTAs sharing one tile's contraction
    bool pair = false, persistent = false, two_tiles = false;
    uint32_t mt_tiles = 16;        // token tile of the shrink's masked-t blocks
    TTiles tt;
};

// flags that pick a form of the tcgen05 kernels (the smallest batches then run on them too)
constexpr uint32_t kTcForms = ATLAS_B200_FLAG_FORCE_TCGEN05 | ATLAS_B200_FLAG_NO_CTA_PAIR | ATLAS_B200_FLAG_NO_K_SPLIT |
                              ATLAS_B200_FLAG_NO_PERSISTENT | ATLAS_B200_FLAG_ONE_TILE_PASS;

// `shrink_tiles`: the shrink of this call can write masked-t tiles
static TcPlan plan_tc(const atlas_b200_linear_desc& d, uint32_t flags, bool shrink_tiles) {
    TcPlan p;
    const bool act_fp4 = (flags & ATLAS_B200_FLAG_ACT_FP4) != 0;
    if (decode_pays(d) && !(flags & (kTcForms | ATLAS_B200_FLAG_ACT_FP4))) {
        p.decode = true;
        return p;
    }
    // Token tile: the smallest power of two that covers m, at most 256 — then halved (down to 64)
    // while the grid would leave more than a quarter of the SMs without a CTA, e.g. for a
    // column shard of a wide layer: more, lighter CTAs finish sooner than few heavy ones.
    p.mt = 16;
    while (p.mt < 256 && p.mt < d.m) p.mt <<= 1;
    const uint32_t f_tiles = (d.n + tc::FT - 1) / tc::FT;
    // Fewer tiles than half the SMs (a decode batch, a column shard): several CTAs share a tile, each
    // contracting a share of K, rather than leaving SMs idle — a CTA's time is set by the weights it has
    // to expand, which only a K split divides.  Clusters of at most 8 CTAs; whole 256-element stages.
    p.k_split = 1;
    p.pair = p.mt >= 128 && !(flags & ATLAS_B200_FLAG_NO_CTA_PAIR);    // pairs of CTAs issue their MMAs together (see tc::Cfg)
    if (!(flags & ATLAS_B200_FLAG_NO_K_SPLIT)) {
        const uint32_t m_tiles = (d.m + p.mt - 1) / p.mt;
        const uint32_t fit = uint32_t(rt_sm_count()) / (f_tiles * m_tiles);
        p.k_split = std::max(1u, std::min(std::min(fit, 8u), d.k / uint32_t(tc::KRAW)));
        // ... but only as many as still lets every cluster be resident at once (a second wave would cost more than the
        // split saves), preferring the shape with pairs, then the one without, then a smaller split
        const bool may_pair = p.pair;
        for (; p.k_split > 1; --p.k_split) {
            if (may_pair && p.k_split <= 4 &&
                tc_active_clusters_of(p.mt, act_fp4, true, p.k_split) >= int(((f_tiles + 1) / 2) * m_tiles)) { p.pair = true; break; }
            if (tc_active_clusters_of(p.mt, act_fp4, false, p.k_split) >= int(f_tiles * m_tiles)) { p.pair = false; break; }
        }
        if (p.k_split == 1) p.pair = may_pair;
    }
    if (p.k_split == 1) {
        while (p.mt > 64 && f_tiles * ((d.m + p.mt - 1) / p.mt) * 4 < uint32_t(rt_sm_count()) * 3) p.mt >>= 1;
        p.pair = p.mt >= 128 && !(flags & ATLAS_B200_FLAG_NO_CTA_PAIR);
    }

    // Masked-t tiles: with scratch to put them in, the shrink writes the activation operand of every LoRA
    // K-step once, in the layout the MMA reads, and the fused kernel's CTAs fetch it by TMA — instead of
    // each CTA rebuilding the same tiles from lora_t.  Needs the strided pool (the TMA producer then feeds
    // both LoRA operands) and the tensor-core shrink; otherwise the in-kernel build stays in use.
    auto tiles_in_ws = [&](uint32_t tile, uint32_t part_rows) {
        TTiles t;
        if (!d.seq_slot || !d.ws || !shrink_tiles) return t;
        const size_t off = act_fp4 ? (act_fp4_ws_bytes(d) + 255) / 256 * 256 : 0;
        const uint32_t cap = std::min(tile, d.max_loras) * ((d.max_rank + 15u) / 16u);
        const size_t rows = size_t((d.m + tile - 1) / tile) * cap * tile;
        if (aligned(d.ws, 256) && d.ws_bytes >= off + rows * 32 && rows < (1ull << 31)) {
            t.tiles = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(d.ws) + off);
            t.cap = cap;
            t.part_rows = part_rows;
        }
        return t;
    };
    p.mt_tiles = p.mt;
    if (b_pool_is_strided(d)) p.tt = tiles_in_ws(p.mt, p.pair ? p.mt / 2 : p.mt);
    // Many tiles per SM pair (a prefill batch): the persistent form, whose operand rings run across tile
    // boundaries and whose row stores overlap the next tile's K loop.  It takes 256-token tiles of CTA pairs
    // without a K split, 16-byte aligned destination rows, and LoRA operands that both come by TMA.
    p.persistent = p.mt == 256 && p.pair && p.k_split == 1 && !(flags & ATLAS_B200_FLAG_NO_PERSISTENT) && d.k % tc::KRAW == 0 &&
                      (!d.seq_slot || b_pool_is_strided(d)) && d.out_row_stride % 8 == 0 &&
                      (d.n_dest ? d.y_col_offset % 8 == 0 : aligned(d.y, 16));
    for (uint32_t r = 0; p.persistent && r < d.n_dest; ++r) p.persistent = aligned(d.y_dest[r], 16);
    // two token tiles of 192 per pass (the expanded weight operand is used twice) where the batch has several passes
    p.two_tiles = p.persistent && !act_fp4 && !(flags & ATLAS_B200_FLAG_ONE_TILE_PASS) && d.m >= 768;
    if (p.two_tiles) {
        // ... unless whole waves say otherwise: the last wave costs a full pass however few CTA pairs it holds, and a pass of two
        // 192-token tiles takes 1.2 (K = 4096) to 1.4 times as long as one of a 256-token tile.  One-tile / two-tile calls by waves, calls
        // with pauses between them (us, K = 4096; K = 14336): 2 : 2 82 / 101; 227 / 310   4 : 3 122 / 131; 364 / 396   5 : 4 133 / 144;
        // 412 / 464   7 : 5 202 / 210; 645 / 675   3 : 2 98 / 98; 276 / 283   25 : 17 658 / 645   2 : 1 60 / 61; 159 / 156.  Call upon
        // call the power limit sets the clock, and two tiles, which expand a weight once for both, need less of it: with 7 : 5 on the
        // other side of the line a layer of 8192 tokens took 2.73 instead of 2.69 ms.  The line lies between 4 : 3 and 7 : 5.
        const int c2 = persist_resident_clusters<192, 2, false>(2), c1 = persist_resident_clusters<256, 1, false>(0);
        if (c1 > 0 && c2 > 0) {
            const uint64_t w2 = (persist_tiles<192, 2>(d) + uint32_t(c2) - 1) / uint32_t(c2);
            const uint64_t w1 = (persist_tiles<256, 1>(d) + uint32_t(c1) - 1) / uint32_t(c1);
            if (w1 * 100 < w2 * 135) p.two_tiles = false;
        }
    }
    if (p.persistent) {
        const int clusters = act_fp4 ? persist_resident_clusters<256, 1, true>(1)
                                     : (p.two_tiles ? persist_resident_clusters<192, 2, false>(2) : persist_resident_clusters<256, 1, false>(0));
        const uint32_t tiles = p.two_tiles ? persist_tiles<192, 2>(d) : persist_tiles<256, 1>(d);
        // (two-tile passes that fit one wave were chosen above because 256-token tiles would take two: 1237 tokens x 4096
        //  features are 64 two-tile passes or 80 tiles on 74 pairs, q_proj 74 -> 38 us)
        p.persistent = clusters > 0 && (p.two_tiles || tiles > uint32_t(clusters));
    }
    if (p.persistent && d.seq_slot) {
        const uint32_t tile = p.two_tiles ? 192u : p.mt;
        const TTiles t = tiles_in_ws(tile, tile / 2);
        p.persistent = t.tiles != nullptr;
        if (t.tiles) { p.tt = t; p.mt_tiles = tile; }
    }
    return p;
}

int nvfp4_lora_linear(const atlas_b200_linear_desc& d, cudaStream_t st, const ShrinkOnly* shrink_only = nullptr) {
    int rc = validate_linear(d);
    if (rc) return rc;
    t_last_variant = ATLAS_B200_VARIANT_NONE;
    if (d.m == 0) return ATLAS_B200_OK;

    const bool staged = (d.flags & ATLAS_B200_FLAG_STAGED_LORA) != 0;
    bool use_tc = !(d.flags & ATLAS_B200_FLAG_FORCE_SIMT) && !staged && tc_eligible(d, false);
    bool reuse_shrink = (d.flags & ATLAS_B200_FLAG_REUSE_SHRINK) != 0;
    if (!use_tc && !staged && !shrink_only && !d.n_dest && !(d.flags & (ATLAS_B200_FLAG_FORCE_SIMT | ATLAS_B200_FLAG_FORCE_TCGEN05 | ATLAS_B200_FLAG_ACT_FP4)) &&
        tc_eligible(d, true)) {
        // These shapes ran on the CUDA cores (64 x 64 tiles of scalar FMAs, then the two-stage LoRA) at a few per cent of this
        // path's rate.  That path computes its shrink on every call, so this one does too.
        use_tc = true;
        reuse_shrink = false;
    }
    if (!use_tc && shrink_only) return ATLAS_B200_ERR_DIMS;
    if (!use_tc && (d.flags & ATLAS_B200_FLAG_FORCE_TCGEN05) && !(d.w_bf16 && !staged && dense_tc_eligible(d))) return ATLAS_B200_ERR_DIMS;
    if (!use_tc && d.n_dest) return ATLAS_B200_ERR_DIMS;          // placement into several buffers is the tcgen05 epilogue's

    const bool act_fp4 = (d.flags & ATLAS_B200_FLAG_ACT_FP4) != 0;
    if (act_fp4) {
        // FP4 activations exist on the tensor-core path only: no other path is substituted for it
        if (!use_tc) return ATLAS_B200_ERR_DIMS;
        if (!d.ws || !aligned(d.ws, 256)) return d.ws ? ATLAS_B200_ERR_ALIGN : ATLAS_B200_ERR_NULL;
        if (d.ws_bytes < act_fp4_ws_bytes(d)) return ATLAS_B200_ERR_WORKSPACE;
        // x -> NVFP4 with a tensor scale of one (scale byte = E4M3 of group max / 6), the activation side
        // of crates/spark-model/src/layers/ops/gemm_fp4.rs:20-40 — unless the caller says they are in place already
        uint8_t* codes = static_cast<uint8_t*>(d.ws);
        if (!(d.flags & ATLAS_B200_FLAG_ACT_FP4_READY) && !shrink_only) {
        const size_t groups = size_t(d.m) * (d.k / 16);
        const unsigned blocks = unsigned(std::min<size_t>((groups + 255) / 256, size_t(rt_sm_count()) * 16));
        rc = launch_chained(quantize_nvfp4_kernel, blocks, 256, st, static_cast<const uint16_t*>(d.x), codes, codes + act_fp4_codes_bytes(d),
                            1.0f, d.m, d.k, d.x_row_stride, 1u);
        if (rc) return rc;
        }
    }
    if (use_tc) {
        ShrinkParams sp{};
        sp.x = static_cast<const uint16_t*>(d.x);
        sp.seq_slot = d.seq_slot;
        sp.a_table = d.a_table;
        sp.b_table = d.b_table;
        sp.scale_table = d.scale_table;
        sp.rank_table = d.rank_table;
        sp.out = static_cast<uint16_t*>(d.lora_t);
        sp.M = d.m; sp.k_in = d.k; sp.max_rank = d.max_rank; sp.x_row_stride = d.x_row_stride; sp.max_loras = d.max_loras;
        sp.a_pool_base = d.a_pool_base; sp.a_slot_stride = d.a_slot_stride;
        sp.post = lora_post(d, act_fp4);

        // (the shrink alone writes tiles, which the decode form does not read: it is planned as a call of the tcgen05 form)
        const TcPlan plan = plan_tc(d, shrink_only ? d.flags | ATLAS_B200_FLAG_FORCE_TCGEN05 : d.flags, shrink_takes_mma_path(sp));
        if (plan.decode) {
            // t rows are written to lora_t by every call of up to eight tokens, and of up to sixteen where N >= 2 K.  Beyond, where calls
            // of the same shape once left tiles in `ws` and were reused, they are read again as the call before has left them.  (Computed
            // again / read, 8 of rank 16: 12 tokens x 4096 x 4096 10.9 / 9.5 us, 16 x 2048 x 4096 10.8 / 7.7.)
            reuse_shrink = reuse_shrink && d.m > 8 && uint64_t(d.n) < 2ull * d.k;
            rc = launch_decode(d, d.seq_slot && !reuse_shrink ? &sp : nullptr, st);
            if (rc == ATLAS_B200_OK) t_last_variant = ATLAS_B200_VARIANT_TCGEN05;
            return rc;
        }
        const TTiles tt = plan.tt;
        if (tt.tiles) {
            sp.tile_out = tt.tiles;
            sp.tile_cap = tt.cap;
            sp.chunk = plan.mt_tiles;
            sp.part_rows = tt.part_rows;
        }
        if (reuse_shrink && (d.flags & kTcForms)) {
            // The call whose result this one is to reuse was made without the form flags: what it left is read only where this
            // form would have left the same.  (It may be rows of lora_t where this one reads tiles — the smallest batches — or
            // tiles of another height.)
            const TcPlan left = plan_tc(d, d.flags & ~kTcForms, shrink_takes_mma_path(sp));
            reuse_shrink = left.tt.tiles == tt.tiles && (!tt.tiles || (left.mt_tiles == plan.mt_tiles && left.tt.part_rows == tt.part_rows));
        }
        if (shrink_only) {
            // the shrink alone, for a row range, into several copies of the scratch: the launch shape decided above fixes
            // the tile layout, exactly as the call that later consumes the tiles (ATLAS_B200_FLAG_REUSE_SHRINK) decides it
            if (!d.seq_slot || !tt.tiles || shrink_only->n_dest == 0 || shrink_only->n_dest > 8) return ATLAS_B200_ERR_DIMS;
            const size_t off = size_t(reinterpret_cast<uint8_t*>(tt.tiles) - static_cast<uint8_t*>(d.ws));
            for (uint32_t i = 0; i < shrink_only->n_dest; ++i)
                if (!shrink_only->ws_dest[i] || !aligned(shrink_only->ws_dest[i], 256)) return ATLAS_B200_ERR_ALIGN;
            sp.tile_out = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(shrink_only->ws_dest[0]) + off);
            for (uint32_t i = 1; i < shrink_only->n_dest; ++i)
                sp.tile_out_more[i - 1] = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(shrink_only->ws_dest[i]) + off);
            sp.n_tile_dest = shrink_only->n_dest;
            sp.m_begin = shrink_only->row_begin;
            sp.m_count = shrink_only->row_count;
            rc = launch_shrink(sp, d.max_loras, st);
            if (rc == ATLAS_B200_OK) t_last_variant = ATLAS_B200_VARIANT_TCGEN05;
            return rc;
        }
        const ShrinkParams* shrink = (d.seq_slot && !reuse_shrink) ? &sp : nullptr;
        if (plan.persistent) {
            if (act_fp4) rc = launch_tc_persist<256, 1, true>(d, 1, shrink, tt, st);
            else if (plan.two_tiles) rc = isolates(d) ? launch_tc_persist<192, 2, false, true>(d, 4, shrink, tt, st) : launch_tc_persist<192, 2, false>(d, 2, shrink, tt, st);
            else rc = isolates(d) ? launch_tc_persist<256, 1, false, true>(d, 3, shrink, tt, st) : launch_tc_persist<256, 1, false>(d, 0, shrink, tt, st);
        } else if (act_fp4) {
            if (plan.mt == 16) rc = launch_tc<16, true, false>(d, 0, shrink, tt, plan.k_split, st);
            else if (plan.mt == 32) rc = launch_tc<32, true, false>(d, 1, shrink, tt, plan.k_split, st);
            else if (plan.mt == 64) rc = launch_tc<64, true, false>(d, 2, shrink, tt, plan.k_split, st);
            else if (plan.mt == 128) rc = plan.pair ? launch_tc<128, true, true>(d, 3, shrink, tt, plan.k_split, st) : launch_tc<128, true, false>(d, 3, shrink, tt, plan.k_split, st);
            else rc = plan.pair ? launch_tc<256, true, true>(d, 4, shrink, tt, plan.k_split, st) : launch_tc<256, true, false>(d, 4, shrink, tt, plan.k_split, st);
        } else if (plan.mt == 16) rc = launch_tc<16, false, false>(d, 0, shrink, tt, plan.k_split, st);
        else if (plan.mt == 32) rc = launch_tc<32, false, false>(d, 1, shrink, tt, plan.k_split, st);
        else if (plan.mt == 64) rc = launch_tc<64, false, false>(d, 2, shrink, tt, plan.k_split, st);
        else if (plan.mt == 128) rc = plan.pair ? launch_tc<128, false, true>(d, 3, shrink, tt, plan.k_split, st) : launch_tc<128, false, false>(d, 3, shrink, tt, plan.k_split, st);
        else rc = plan.pair ? launch_tc<256, false, true>(d, 4, shrink, tt, plan.k_split, st) : launch_tc<256, false, false>(d, 4, shrink, tt, plan.k_split, st);
        if (rc == ATLAS_B200_OK) t_last_variant = ATLAS_B200_VARIANT_TCGEN05;
        return rc;
    }

    // Base linear — a dense BF16 weight on the tensor cores where the shape allows, everything else on CUDA cores —
    // then the reference's two-stage LoRA in place
    const bool dense_tc = !(d.flags & ATLAS_B200_FLAG_FORCE_SIMT) && !staged && dense_tc_eligible(d);
    // The shrink goes first where the base can run beside it: it waits for what is before the call, and the base then starts at once.
    // That is where its grid is resident at once, and for few tokens and features.  Base first / shrink first (us), adapters x rank:
    // 4096 x 4096, 16 tokens 4 x 16 19.6 / 14.2, 64 x 64 23.2 / 20.7, 100 tokens 128 x 16 35.8 / 30.3, 64 x 64 45.6 / 48.0, 300 tokens
    // 128 x 16 50.6 / 54.2, 8 x 64 46.4 / 45.9, 1000 tokens 4 x 16 65.1 / 65.5, 8 x 64 89.7 / 95.6; 14336 x 4096, 64 tokens 4 x 16 42.7 /
    // 40.8, 64 x 64 71.9 / 81.8; 1024 x 8192, 512 tokens 8 x 64 49.1 / 43.3, 64 x 64 78.7 / 87.1, 1000 tokens 4 x 16 51.0 / 41.1, 1500
    // tokens 59.8 / 66.9.
    const uint64_t shrink_ctas = uint64_t(d.max_loras) * ((d.max_rank + 15) / 16) * ((d.m + SHM_CHUNK - 1) / SHM_CHUNK) * SHM_KSPLIT;
    const bool shrink_first = dense_tc && d.seq_slot && d.m <= 1024 &&
                              (shrink_ctas <= uint64_t(rt_sm_count()) * MMA_SHRINK_CTAS_PER_SM || (d.m <= 64 && d.n <= 4096));
    auto base = [&]() { return dense_tc ? launch_dense_tc(d, shrink_first, st) : launch_simt_linear(d, st); };
    if (!shrink_first) {
        rc = base();
        if (rc) return rc;
    }
    if (d.seq_slot) {
        ShrinkParams sp{};
        sp.x = static_cast<const uint16_t*>(d.x);
        sp.seq_slot = d.seq_slot;
        sp.a_table = d.a_table;
        sp.b_table = d.b_table;
        sp.rank_table = d.rank_table;
        sp.out = static_cast<uint16_t*>(d.lora_t);
        sp.M = d.m; sp.k_in = d.k; sp.max_rank = d.max_rank; sp.x_row_stride = d.x_row_stride; sp.max_loras = d.max_loras;
        sp.post = 0.0f;
        rc = launch_shrink(sp, d.max_loras, st, shrink_first ? MachineBeside::all : MachineBeside::none);
        if (rc) return rc;
        if (shrink_first) {
            rc = base();
            if (rc) return rc;
        }
        ExpandParams ep{};
        ep.xa = static_cast<const uint16_t*>(d.lora_t);
        ep.seq_slot = d.seq_slot;
        ep.a_table = d.a_table;
        ep.b_table = d.b_table;
        ep.scale_table = d.scale_table;
        ep.out = static_cast<uint16_t*>(d.y);
        ep.M = d.m; ep.n_out = d.n; ep.max_rank = d.max_rank; ep.out_row_stride = d.out_row_stride; ep.max_loras = d.max_loras;
        rc = launch_expand(ep, st);
        if (rc) return rc;
    }
    t_last_variant = dense_tc ? ATLAS_B200_VARIANT_TCGEN05 : ATLAS_B200_VARIANT_SIMT;
    return ATLAS_B200_OK;
}

}  // namespace ops
}  // namespace atlas

// =============================================================================================
// extern "C"
// =============================================================================================
using namespace atlas;

extern "C" {

int atlas_b200_lora_bgmv(const void* x, const int32_t* seq_slot, const uint64_t* a_table, const uint64_t* b_table,
                         const float* scale_table, void* base_out, void* lora_xa, uint32_t n, uint32_t k_in,
                         uint32_t n_out, uint32_t max_rank, uint32_t x_row_stride, uint32_t out_row_stride,
                         uint32_t max_loras, void* stream) {
    return ops::apply_lora_bgmv(x, seq_slot, a_table, b_table, scale_table, base_out, lora_xa, n, k_in, n_out, max_rank,
                                x_row_stride, out_row_stride, max_loras, static_cast<cudaStream_t>(stream));
}

int atlas_b200_lora_delta(const void* x, const void* a, const void* b, float scale, void* base_out, void* lora_xa,
                          void* lora_delta, uint32_t m, uint32_t k_in, uint32_t n_out, uint32_t max_rank, void* stream) {
    return ops::apply_lora_delta(x, a, b, scale, base_out, lora_xa, lora_delta, m, k_in, n_out, max_rank,
                                 static_cast<cudaStream_t>(stream));
}

int atlas_b200_w4a16_gemm(const void* a_bf16, const void* b_packed, const void* b_scale, float scale2, void* c_bf16,
                          uint32_t m, uint32_t n, uint32_t k, void* ws, size_t ws_bytes, void* stream) {
    (void)ws; (void)ws_bytes;
    atlas_b200_linear_desc d;
    std::memset(&d, 0, sizeof(d));
    d.x = a_bf16; d.m = m; d.k = k; d.x_row_stride = k;
    d.n = n; d.w_packed = b_packed; d.w_scale = b_scale; d.scale2 = scale2;
    d.y = c_bf16; d.out_row_stride = n;
    return ops::nvfp4_lora_linear(d, static_cast<cudaStream_t>(stream));
}

int atlas_b200_dequant_nvfp4_to_bf16(const void* packed, const void* scales, void* out_bf16, float combined_global,
                                     uint32_t n, uint32_t k, void* stream) {
    if (n == 0 || k == 0) return ATLAS_B200_OK;
    if (!packed || !scales || !out_bf16) return ATLAS_B200_ERR_NULL;
    if (k % 16 != 0) return ATLAS_B200_ERR_DIMS;
    if (!aligned(out_bf16, 4)) return ATLAS_B200_ERR_ALIGN;
    const size_t groups = size_t(n) * (k / 16);
    const unsigned blocks = unsigned(std::min<size_t>((groups + 255) / 256, size_t(rt_sm_count()) * 16));
    dequant_nvfp4_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(packed), static_cast<const uint8_t*>(scales), static_cast<uint16_t*>(out_bf16),
        combined_global, groups, aligned(packed, 8) && aligned(out_bf16, 16) ? 1u : 0u);
    return launch_status();
}

int atlas_b200_quantize_bf16_to_nvfp4(const void* in_bf16, void* packed, void* scales, float scale2, uint32_t n,
                                      uint32_t k, void* stream) {
    if (n == 0 || k == 0) return ATLAS_B200_OK;
    if (!in_bf16 || !packed || !scales) return ATLAS_B200_ERR_NULL;
    if (k % 16 != 0) return ATLAS_B200_ERR_DIMS;
    const size_t groups = size_t(n) * (k / 16);
    const unsigned blocks = unsigned(std::min<size_t>((groups + 255) / 256, size_t(rt_sm_count()) * 16));
    const uint32_t vec = aligned(in_bf16, 16) && aligned(packed, 8) && k % 16 == 0;
    return launch_chained(quantize_nvfp4_kernel, blocks, 256, static_cast<cudaStream_t>(stream),
        static_cast<const uint16_t*>(in_bf16), static_cast<uint8_t*>(packed), static_cast<uint8_t*>(scales), scale2, n, k, k, vec);
}

int atlas_b200_nvfp4_global_absmax(const void* in_bf16, float* global_max_dev, size_t total, void* stream) {
    if (total == 0) return ATLAS_B200_OK;
    if (!in_bf16 || !global_max_dev) return ATLAS_B200_ERR_NULL;
    if (!aligned(in_bf16, 2) || !aligned(global_max_dev, 4)) return ATLAS_B200_ERR_ALIGN;
    const unsigned blocks = unsigned(std::min<size_t>((total / 8 + 255) / 256 + 1, size_t(rt_sm_count()) * 8));
    nvfp4_global_absmax_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint16_t*>(in_bf16), global_max_dev, total);
    return launch_status();
}

float atlas_b200_nvfp4_scale2_from_absmax(float global_max) { return global_max / (6.0f * 448.0f); }

float atlas_b200_nvfp4_combined_global_scale(float stored_scale, int is_reciprocal) {
    if (!is_reciprocal) return stored_scale;
    return stored_scale != 0.0f ? 1.0f / stored_scale : 0.0f;
}

int atlas_b200_push_columns(const void* src, uint32_t src_row_stride, void* const* dest, uint32_t n_dest, uint32_t dst_row_stride,
                            uint32_t m, uint32_t n_cols, void* stream) {
    if (!src || (!dest && n_dest)) return ATLAS_B200_ERR_NULL;
    if (n_dest > uint32_t(PUSH_MAX_DEST)) return ATLAS_B200_ERR_LIMIT;
    if (m == 0 || n_cols == 0 || n_dest == 0) return ATLAS_B200_OK;
    if (n_cols > src_row_stride || n_cols > dst_row_stride) return ATLAS_B200_ERR_DIMS;
    if (n_cols % 8 || src_row_stride % 8 || dst_row_stride % 8 || !aligned(src, 16)) return ATLAS_B200_ERR_ALIGN;
    PushParams p{};
    p.src = static_cast<const uint4*>(src);
    for (uint32_t d = 0; d < n_dest; ++d) {
        if (!dest[d]) return ATLAS_B200_ERR_NULL;
        if (!aligned(dest[d], 16)) return ATLAS_B200_ERR_ALIGN;
        p.dst[d] = static_cast<uint4*>(dest[d]);
    }
    p.n_dest = n_dest;
    p.m = m;
    p.chunks_per_row = n_cols / 8;
    p.src_row_chunks = src_row_stride / 8;
    p.dst_row_chunks = dst_row_stride / 8;
    const uint64_t total = uint64_t(m) * p.chunks_per_row;
    const uint64_t want = (total + uint64_t(PUSH_THREADS) * 4 - 1) / (uint64_t(PUSH_THREADS) * 4);
    const uint32_t grid = uint32_t(std::min<uint64_t>(std::max<uint64_t>(want, 1), uint64_t(rt_sm_count()) * 2));
    // same shared-memory carve-out as the tcgen05 kernels: an SM must not have to drain and be reconfigured before it can
    // take one of these CTAs next to theirs
    DeviceState* dst_state = device_state();
    if (dst_state && !dst_state->push_attr_set) {
        cudaFuncSetAttribute(push_columns_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        dst_state->push_attr_set = true;
    }
    push_columns_kernel<<<grid, PUSH_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(p);
    return launch_status();
}

static int kv_norm_rope_cache_write(const void* k_in, const void* v_in, uint32_t in_row_stride, const void* k_norm_weight,
                                    const uint32_t* positions, const uint32_t* positions_h, const uint32_t* positions_w, const long long* slot_mapping, void* k_cache, void* v_cache,
                                        uint32_t tokens, uint32_t kv_heads, uint32_t head_dim, uint32_t rotary_dim, uint32_t block_size,
                                        float rms_eps, float theta, void* stream, float fp8_inv_scale = 0.0f) {
    if (!k_in || !k_norm_weight || !positions || !slot_mapping || !k_cache || (v_in && !v_cache)) return ATLAS_B200_ERR_NULL;
    if (tokens == 0 || kv_heads == 0) return ATLAS_B200_OK;
    if (head_dim == 0 || head_dim % 32 || head_dim > uint32_t(KVE_MAX_HEAD_DIM) || rotary_dim > head_dim || rotary_dim % 64 ||
        block_size == 0 || in_row_stride < kv_heads * head_dim)
        return ATLAS_B200_ERR_DIMS;
    KvEpilogueParams p{};
    p.k_in = static_cast<const uint16_t*>(k_in);
    p.v_in = static_cast<const uint16_t*>(v_in);
    p.k_norm_w = static_cast<const uint16_t*>(k_norm_weight);
    p.positions = positions;
    p.positions_h = positions_h;
    p.positions_w = positions_w;
    p.slot_mapping = slot_mapping;
    p.k_cache = static_cast<uint16_t*>(k_cache);
    p.v_cache = static_cast<uint16_t*>(v_cache);
    p.tokens = tokens; p.kv_heads = kv_heads; p.head_dim = head_dim; p.rotary_dim = rotary_dim; p.block_size = block_size;
    p.in_row_stride = in_row_stride; p.rms_eps = rms_eps; p.theta = theta; p.fp8_inv_scale = fp8_inv_scale;
    const dim3 grid((tokens + KVE_TOKENS - 1) / KVE_TOKENS), block(KVE_WARPS * 32);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool exact = rotary_dim == 64 && fp8_inv_scale == 0.0f && (head_dim == 64 || head_dim == 128 || head_dim == 256);
    if (head_dim <= 64) return exact ? launch_chained(kv_norm_rope_cache_kernel<2, true>, grid, block, st, p) : launch_chained(kv_norm_rope_cache_kernel<2, false>, grid, block, st, p);
    if (head_dim <= 128) return exact ? launch_chained(kv_norm_rope_cache_kernel<4, true>, grid, block, st, p) : launch_chained(kv_norm_rope_cache_kernel<4, false>, grid, block, st, p);
    return exact ? launch_chained(kv_norm_rope_cache_kernel<8, true>, grid, block, st, p) : launch_chained(kv_norm_rope_cache_kernel<8, false>, grid, block, st, p);
}

int atlas_b200_kv_norm_rope_cache_write(const void* k_in, const void* v_in, uint32_t in_row_stride, const void* k_norm_weight,
                                        const uint32_t* positions, const long long* slot_mapping, void* k_cache, void* v_cache,
                                        uint32_t tokens, uint32_t kv_heads, uint32_t head_dim, uint32_t rotary_dim, uint32_t block_size,
                                        float rms_eps, float theta, void* stream) {
    return kv_norm_rope_cache_write(k_in, v_in, in_row_stride, k_norm_weight, positions, nullptr, nullptr, slot_mapping, k_cache, v_cache, tokens,
                                    kv_heads, head_dim, rotary_dim, block_size, rms_eps, theta, stream);
}

int atlas_b200_k_norm_rope_cache_write_fp8(const void* k_in, uint32_t in_row_stride, const void* k_norm_weight, const uint32_t* positions,
                                           const long long* slot_mapping, void* k_cache_fp8, uint32_t tokens, uint32_t kv_heads,
                                           uint32_t head_dim, uint32_t rotary_dim, uint32_t block_size, float rms_eps, float theta,
                                           float inv_scale, void* stream) {
    if (!(inv_scale > 0.0f)) return ATLAS_B200_ERR_DIMS;
    return kv_norm_rope_cache_write(k_in, nullptr, in_row_stride, k_norm_weight, positions, nullptr, nullptr, slot_mapping, k_cache_fp8, nullptr,
                                    tokens, kv_heads, head_dim, rotary_dim, block_size, rms_eps, theta, stream, inv_scale);
}

int atlas_b200_kv_norm_mrope_cache_write(const void* k_in, const void* v_in, uint32_t in_row_stride, const void* k_norm_weight,
                                         const uint32_t* pos_t, const uint32_t* pos_h, const uint32_t* pos_w, const long long* slot_mapping,
                                         void* k_cache, void* v_cache, uint32_t tokens, uint32_t kv_heads, uint32_t head_dim,
                                         uint32_t rotary_dim, uint32_t block_size, float rms_eps, float theta, void* stream) {
    if (!pos_h || !pos_w) return ATLAS_B200_ERR_NULL;
    return kv_norm_rope_cache_write(k_in, v_in, in_row_stride, k_norm_weight, pos_t, pos_h, pos_w, slot_mapping, k_cache, v_cache, tokens,
                                    kv_heads, head_dim, rotary_dim, block_size, rms_eps, theta, stream);
}

int atlas_b200_qkv_norm_rope_cache_write(void* q, const void* k_in, const void* v_in, uint32_t q_row_stride, uint32_t kv_row_stride,
                                         const void* q_norm_weight, const void* k_norm_weight, const uint32_t* positions,
                                         const float* inv_freq, const long long* slot_mapping, void* k_cache, void* v_cache,
                                         uint32_t tokens, uint32_t q_heads, uint32_t kv_heads, uint32_t head_dim, uint32_t rotary_dim,
                                         uint32_t block_size, float rms_eps, float attention_factor, int norm_offset_one, void* stream) {
    if (!q || !k_in || !v_in || !q_norm_weight || !k_norm_weight || !positions || !slot_mapping || !k_cache || !v_cache ||
        (rotary_dim && !inv_freq))
        return ATLAS_B200_ERR_NULL;
    if (tokens == 0 || q_heads + kv_heads == 0) return ATLAS_B200_OK;
    if (head_dim == 0 || head_dim % 2 || head_dim > uint32_t(KVE_MAX_HEAD_DIM) || rotary_dim > head_dim || rotary_dim % 2 ||
        block_size == 0 || q_row_stride < q_heads * head_dim || kv_row_stride < kv_heads * head_dim)
        return ATLAS_B200_ERR_DIMS;
    // packed pairs are read as 32-bit words
    if (!aligned(q, 4) || !aligned(k_in, 4) || !aligned(v_in, 4) || !aligned(v_cache, 4) || !aligned(q_norm_weight, 4) ||
        !aligned(k_norm_weight, 4) || q_row_stride % 2 || kv_row_stride % 2)
        return ATLAS_B200_ERR_ALIGN;
    QkvEpilogueParams p{};
    p.q = static_cast<uint16_t*>(q);
    p.k_in = static_cast<const uint16_t*>(k_in);
    p.v_in = static_cast<const uint16_t*>(v_in);
    p.q_norm_w = static_cast<const uint16_t*>(q_norm_weight);
    p.k_norm_w = static_cast<const uint16_t*>(k_norm_weight);
    p.positions = positions; p.inv_freq = inv_freq; p.slot_mapping = slot_mapping;
    p.k_cache = static_cast<uint16_t*>(k_cache);
    p.v_cache = static_cast<uint16_t*>(v_cache);
    p.tokens = tokens; p.q_heads = q_heads; p.kv_heads = kv_heads; p.head_dim = head_dim; p.rotary_dim = rotary_dim;
    p.block_size = block_size; p.q_row_stride = q_row_stride; p.kv_row_stride = kv_row_stride;
    p.rms_eps = rms_eps; p.attention_factor = attention_factor; p.norm_offset_one = norm_offset_one ? 1u : 0u;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool exact = rotary_dim == 64 && (head_dim == 64 || head_dim == 128 || head_dim == 256);
    if (head_dim <= 64) return exact ? launch_chained(qkv_norm_rope_cache_kernel<1, true>, tokens, KVE_WARPS * 32, st, p)
                              : launch_chained(qkv_norm_rope_cache_kernel<1, false>, tokens, KVE_WARPS * 32, st, p);
    if (head_dim <= 128) return exact ? launch_chained(qkv_norm_rope_cache_kernel<2, true>, tokens, KVE_WARPS * 32, st, p)
                                    : launch_chained(qkv_norm_rope_cache_kernel<2, false>, tokens, KVE_WARPS * 32, st, p);
    return exact ? launch_chained(qkv_norm_rope_cache_kernel<4, true>, tokens, KVE_WARPS * 32, st, p)
               : launch_chained(qkv_norm_rope_cache_kernel<4, false>, tokens, KVE_WARPS * 32, st, p);
}

int atlas_b200_copy_columns(const void* src, uint32_t src_row_stride, void* const* dest, uint32_t n_dest, uint32_t dst_row_stride,
                            uint32_t m, uint32_t n_cols, void* stream) {
    if (!src || (!dest && n_dest)) return ATLAS_B200_ERR_NULL;
    if (m == 0 || n_cols == 0 || n_dest == 0) return ATLAS_B200_OK;
    if (n_cols > src_row_stride || n_cols > dst_row_stride) return ATLAS_B200_ERR_DIMS;
    for (uint32_t d = 0; d < n_dest; ++d) {
        if (!dest[d]) return ATLAS_B200_ERR_NULL;
        // one strided copy per destination, carried by the copy engines
        cudaError_t e = cudaMemcpy2DAsync(dest[d], size_t(dst_row_stride) * 2, src, size_t(src_row_stride) * 2, size_t(n_cols) * 2, m,
                                          cudaMemcpyDeviceToDevice, static_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return cuda_status(e);
    }
    return ATLAS_B200_OK;
}

int atlas_b200_silu_mul(const void* gate_bf16, const void* up_bf16, void* out_bf16, float gate_scale, float up_scale, float swiglu_limit,
                        uint32_t m, uint32_t k, uint32_t in_row_stride, uint32_t out_row_stride, void* stream) {
    if (m == 0 || k == 0) return ATLAS_B200_OK;
    if (!gate_bf16 || !up_bf16 || !out_bf16) return ATLAS_B200_ERR_NULL;
    if (k % 8 != 0 || in_row_stride < k || out_row_stride < k) return ATLAS_B200_ERR_DIMS;
    if (in_row_stride % 8 != 0 || out_row_stride % 8 != 0 || !aligned(gate_bf16, 16) || !aligned(up_bf16, 16) || !aligned(out_bf16, 16))
        return ATLAS_B200_ERR_ALIGN;
    const size_t vecs = size_t(m) * (k / 8);
    const unsigned blocks = unsigned(std::min<size_t>((vecs + 255) / 256, size_t(rt_sm_count()) * 16));
    return launch_chained(silu_mul_kernel, blocks, 256, static_cast<cudaStream_t>(stream), 
        static_cast<const uint16_t*>(gate_bf16), static_cast<const uint16_t*>(up_bf16), static_cast<uint16_t*>(out_bf16), gate_scale,
        up_scale, swiglu_limit, m, k, in_row_stride, out_row_stride);
}

int atlas_b200_silu_mul_quant_nvfp4(const void* gate_bf16, const void* up_bf16, void* ws, size_t ws_bytes, float gate_scale, float up_scale,
                                    float swiglu_limit, uint32_t m, uint32_t k, uint32_t in_row_stride, void* stream) {
    if (m == 0 || k == 0) return ATLAS_B200_OK;
    if (!gate_bf16 || !up_bf16 || !ws) return ATLAS_B200_ERR_NULL;
    if (k % 16 != 0 || in_row_stride < k) return ATLAS_B200_ERR_DIMS;
    if (in_row_stride % 8 != 0 || !aligned(gate_bf16, 16) || !aligned(up_bf16, 16) || !aligned(ws, 256)) return ATLAS_B200_ERR_ALIGN;
    const size_t codes_bytes = (size_t(m) * (k / 2) + 255) / 256 * 256;
    if (ws_bytes < codes_bytes + size_t(m) * (k / 16)) return ATLAS_B200_ERR_WORKSPACE;
    const size_t groups = size_t(m) * (k / 16);
    const unsigned blocks = unsigned(std::min<size_t>((groups + 255) / 256, size_t(rt_sm_count()) * 16));
    uint8_t* codes = static_cast<uint8_t*>(ws);
    return launch_chained(silu_mul_quant_nvfp4_kernel, blocks, 256, static_cast<cudaStream_t>(stream), 
        static_cast<const uint16_t*>(gate_bf16), static_cast<const uint16_t*>(up_bf16), codes, codes + codes_bytes, gate_scale, up_scale,
        swiglu_limit, m, k, in_row_stride);
}

int atlas_b200_nvfp4_lora_linear(const atlas_b200_linear_desc* desc, void* stream) {
    if (!desc) return ATLAS_B200_ERR_NULL;
    return ops::nvfp4_lora_linear(*desc, static_cast<cudaStream_t>(stream));
}

int atlas_b200_lora_shrink_tiles(const atlas_b200_linear_desc* desc, uint32_t row_begin, uint32_t row_count,
                                 void* const* ws_dest, uint32_t n_dest, void* stream) {
    if (!desc || !ws_dest) return ATLAS_B200_ERR_NULL;
    ops::ShrinkOnly so{row_begin, row_count, n_dest, ws_dest};
    return ops::nvfp4_lora_linear(*desc, static_cast<cudaStream_t>(stream), &so);
}

// ---------------------------------------------------------------------------------------------
// Fused layer for callers that cannot allocate device memory.
//
// Some hosts of this library may launch kernels but may not call cudaMalloc: a plug-in that is
// handed tensors by an engine which owns every byte of device memory, or code running inside a
// region (a captured serving step, a real-time loop) where the allocator must not be entered.
// Such a caller has nowhere to get the shrink scratch `lora_t` from.  This entry point keeps that
// scratch in a fixed array inside the library image instead, so the caller passes inputs and the
// output only.
//
// The array holds ATLAS_B200_STATIC_SCRATCH_ELEMS BF16 values (1 MiB) on every GPU that loads the
// library, for the life of the process.  A call needs m * max_rank of them; more is refused.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) uint16_t g_static_lora_t[ATLAS_B200_STATIC_SCRATCH_ELEMS];

namespace atlas {
// In host code `g_static_lora_t` names a host-side shadow of the symbol, not device memory, so the
// device address is asked for once per device, with that device current, and cached.
static void* g_static_scratch_addr[kMaxDevices] = {};
static std::mutex g_static_scratch_mutex;

static int static_scratch_for_current_device(void** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e);
    if (dev < 0 || dev >= kMaxDevices) return ATLAS_B200_ERR_LIMIT;
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (!g_static_scratch_addr[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_lora_t);
        if (e != cudaSuccess) return cuda_status(e);
        if (!ptr) return ATLAS_B200_ERR_NULL;
        g_static_scratch_addr[dev] = ptr;
    }
    *out = g_static_scratch_addr[dev];
    return ATLAS_B200_OK;
}
}  // namespace atlas

extern "C" int atlas_b200_nvfp4_lora_linear_noalloc(const atlas_b200_linear_desc* desc, void* stream) {
    if (!desc) return ATLAS_B200_ERR_NULL;
    atlas_b200_linear_desc d = *desc;
    if (d.seq_slot) {
        // validate the size before anything else so that an oversized call never touches the array
        if (d.max_rank == 0 || d.max_loras == 0) return ATLAS_B200_ERR_DIMS;
        if (uint64_t(d.m) * uint64_t(d.max_rank) > uint64_t(ATLAS_B200_STATIC_SCRATCH_ELEMS)) return ATLAS_B200_ERR_LIMIT;
        void* scratch = nullptr;
        const int rc = static_scratch_for_current_device(&scratch);
        if (rc) return rc;
        // Nothing in the scratch has to start at zero: the shrink writes every element of every routed
        // row (pad ranks as zeros) and un-routed rows are never read, so leftovers of an earlier call
        // are harmless and no clearing pass is launched.
        d.lora_t = scratch;
    }
    return ops::nvfp4_lora_linear(d, static_cast<cudaStream_t>(stream));
}

int atlas_b200_device_status(uint32_t* out_word, int clear) {
    if (!out_word) return ATLAS_B200_ERR_NULL;
    cudaError_t e = cudaMemcpyFromSymbol(out_word, g_status_word, sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_status(e);
    if (clear) {
        const uint32_t zero = 0;
        e = cudaMemcpyToSymbol(g_status_word, &zero, sizeof(uint32_t));
    }
    return cuda_status(e);
}

int atlas_b200_selftest_bounded_wait(uint64_t limit_ns, uint32_t out_host[3]) {
    if (!out_host) return ATLAS_B200_ERR_NULL;
    if (limit_ns == 0 || limit_ns > 100000000ull) return ATLAS_B200_ERR_LIMIT;        // at most 0.1 s: this is a test of giving up
    uint32_t* out_dev = nullptr;
    cudaError_t e = cudaMalloc(&out_dev, 3 * sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_status(e);
    cudaMemset(out_dev, 0xFF, 3 * sizeof(uint32_t));
    tc::bounded_wait_selftest_kernel<<<1, 64>>>(limit_ns, uint32_t(STATUS_WAIT_EXPIRED_PRODUCER), out_dev);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out_host, out_dev, 3 * sizeof(uint32_t), cudaMemcpyDeviceToHost);
    cudaFree(out_dev);
    return cuda_status(e);
}

int atlas_b200_selftest_ring_wait(uint32_t* out_written) {
    if (!out_written) return ATLAS_B200_ERR_NULL;
    constexpr uint32_t K = 1024, N = 16;
    using R = DcmRing<1, 8>;
    const auto kernel = nvfp4_lora_decode_mma_kernel<1, 1, 8, true, true, true>;
    uint16_t* buf = nullptr;                                  // x [K], then y [N]
    uint16_t y[N];
    CUtensorMap none;
    std::memset(&none, 0, sizeof(none));                      // never dereferenced: nothing is fetched
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM_BYTES);
    if (e == cudaSuccess) e = cudaMalloc(&buf, (K + N) * sizeof(uint16_t));
    if (e != cudaSuccess) return cuda_status(e);
    e = cudaMemset(buf, 0x5A, (K + N) * sizeof(uint16_t));
    tc::Params p{};
    DecodeParams w{};
    w.x = buf; w.x_row_stride = K;
    p.y = p.y_dest[0] = buf + K; p.n_dest = 1;
    p.M = 1; p.N = N; p.K = K; p.out_row_stride = N; p.out_scale = 1.0f; p.k_split = 1;
    if (e == cudaSuccess) {
        kernel<<<1, 32 * 9, R::SMEM_BYTES>>>(w, p, none, none);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(y, buf + K, sizeof(y), cudaMemcpyDeviceToHost);
    cudaFree(buf);
    *out_written = 0;
    for (const uint16_t v : y) *out_written += v != 0x5A5A;
    return cuda_status(e);
}

int atlas_b200_last_variant(void) { return t_last_variant; }

int atlas_b200_last_launch_shape(uint32_t out[4]) {
    if (!out) return ATLAS_B200_ERR_NULL;
    for (int i = 0; i < 4; ++i) out[i] = t_last_shape[i];
    return ATLAS_B200_OK;
}

int atlas_b200_last_persistent_shape(uint32_t out[2]) {
    if (!out) return ATLAS_B200_ERR_NULL;
    out[0] = t_last_shape[4];
    out[1] = t_last_shape[5];
    return ATLAS_B200_OK;
}

int atlas_b200_last_launch_details(uint32_t out[2]) {
    if (!out) return ATLAS_B200_ERR_NULL;
    out[0] = t_last_shape[6];
    out[1] = t_last_shape[7];
    return ATLAS_B200_OK;
}

int atlas_b200_set_profile_buffer(void* device_buffer, size_t n_words) {
    g_profile_buf = static_cast<unsigned long long*>(device_buffer);
    g_profile_words = device_buffer ? n_words : 0;
    return ATLAS_B200_OK;
}

const char* atlas_b200_version(void) { return "atlas_b200 0.1 (sm_100a)"; }

}  // extern "C"
