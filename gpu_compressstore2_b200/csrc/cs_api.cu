// cs_api.cu — the C ABI (include/compressstore.h): argument checking, workspace layout,
// algorithm resolution, the per-(device, stream) scratch cache of the plain call, and the
// generator / pass entry points.
#include <atomic>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include <cuda_runtime.h>

#include "compressstore.h"
#include "cs_internal.cuh"
#include "cs_tuning.h"

namespace cs {

static std::atomic<uint64_t> g_launches{0};
void note_launch(uint64_t k)
{
    g_launches.fetch_add(k, std::memory_order_relaxed);
}

namespace {

constexpr uint64_t MAX_N = (1ull << 40) - 1; // status words carry 40-bit offsets
// The TMA 1-pass kernel takes one-tile units for a column with fewer full units than SMs and at most this many
// one-tile units (the workspace reserves statuses for that many). Such columns run in slices unless skip = 2
// asks for whole tiles.
constexpr uint64_t SHORT_UNITS_MAX = 1024;
// ... and the deeper payload ring (mode 2) for 4- and 8-byte columns of at least this many
// full units per SM.
constexpr uint64_t DEEP_UNITS_PER_SM = 16;
// Most slices per SM for which a 1-pass call of 4- and 8-byte elements runs in slices (cs_slices.cu)
// rather than through the TMA kernel; 1- and 2-byte columns of any length do. Per call on B200, inputs
// from HBM, TMA / slices, us: u32 2^20 8.7 / 5.3, 2^22 13.7 / 9.1; by slices per SM
//   u32       8            12           13           13.8         15           16           18           24
//   p = 0.01  16.2 / 10.6  19.4 / 14.2  19.7 / 14.5  20.0 / 15.4  22.3 / 17.0  22.7 / 17.5  24.3 / 20.1  29.2 / 26.3
//   p = 0.1   16.9 / 14.9  20.4 / 19.3  20.8 / 19.6  21.1 / 21.7  23.5 / 22.6  23.8 / 22.8  25.9 / 26.1  30.8 / 32.9
//   p = 0.5   18.6 / 17.6  24.4 / 22.5  24.7 / 23.2  24.9 / 25.5  28.2 / 26.7  29.0 / 27.1  32.4 / 30.7  39.2 / 38.1
//   p = 0.9   21.3 / 20.4  28.0 / 25.8  28.6 / 27.1  29.2 / 29.2  33.5 / 30.6  34.3 / 31.4  38.2 / 35.3  49.3 / 44.5
//   u64       6            7            8            9            10           12           14
//   p = 0.1   14.0 / 11.4  16.4 / 15.4  16.0 / 16.8  16.4 / 17.7  16.8 / 18.3  19.4 / 19.7  19.9 / 22.7
//   p = 0.5   15.3 / 13.3  18.0 / 15.6  17.6 / 16.8  18.6 / 17.6  19.6 / 19.2  23.7 / 21.7  24.6 / 24.8
// Both kernels step, the slices where an SM's last turn takes a second CTA, the TMA kernel by half units, and where
// the call's status words fall in memory moves either by several per cent: 13.8 per SM at 0.1 over 24 places TMA
// 20.7 .. 25.2, mean 21.4, slices 21.2 .. 22.2, mean 21.65; at 0.5 25.4 and 25.5. u8 2^24 16.5 / 11.3, 2^28 135 / 103;
// u16 2^24 21.6 / 18.3, 2^26 51.6 / 48.
constexpr uint64_t slices_per_sm(uint32_t elem_bytes)
{
    return elem_bytes == 4 ? 18 : 8;
}
// Sparse 16K-element items from which on a column without the block pass may be gathered, as many as the block
// pass asks for.
constexpr uint64_t GATHER_ITEMS_MIN = 256;
constexpr uint64_t DEFAULT_TIMEOUT_NS = 2000000000ull;

struct DeviceInfo {
    int sms = 0;
    int major = 0;
};

std::mutex g_dev_mu;
std::map<int, DeviceInfo> g_dev;

int current_device_info(DeviceInfo* out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    {
        std::lock_guard<std::mutex> lk(g_dev_mu);
        auto it = g_dev.find(dev);
        if (it != g_dev.end()) {
            *out = it->second;
            return CS_SUCCESS;
        }
    }
    DeviceInfo di;
    if (cudaDeviceGetAttribute(&di.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    if (cudaDeviceGetAttribute(&di.major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    if (di.major != 10) return CS_ERR_NO_DEVICE; // built for sm_100a only
    std::lock_guard<std::mutex> lk(g_dev_mu);
    g_dev[dev] = di;
    *out = di;
    return CS_SUCCESS;
}

inline size_t align256(size_t x)
{
    return (x + 255) & ~static_cast<size_t>(255);
}

inline bool is_pow2(uint64_t x)
{
    return x && !(x & (x - 1));
}

inline uint32_t ilog2(uint64_t x)
{
    uint32_t r = 0;
    while ((1ull << r) < x) ++r;
    return r;
}

inline bool aligned(const void* p, uintptr_t a)
{
    return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0;
}

struct Layout {
    uint64_t num_tiles = 0;   // units (UNIT_TILES tiles) of the TMA kernel
    uint64_t num_units1 = 0;  // one-tile units of the 1-pass kernel for short columns
    uint64_t num_chunks = 0;  // popcount chunks
    uint64_t scan_tiles = 0;  // look-back scan tiles over the chunks
    size_t off_status = 0;
    size_t off_scan_status = 0;
    size_t off_counts = 0;
    size_t off_offsets = 0;
    size_t off_blk_base = 0;  // per-2^18-element block prefixes of the reduce-then-scan pass
    size_t off_item_flags = 0; // sparse items of the hybrid writeout, marked by pass 1
    size_t off_flags = 0;     // pass 1's per-CTA sparse flags
    size_t total = 0;
};

// All regions every algorithm may need, so AUTO may switch algorithm freely.
Layout plan_layout(uint64_t n, uint32_t elem_bytes, uint32_t chunk_log2)
{
    Layout l;
    const uint64_t ue = unit_elems_for(elem_bytes);
    const uint64_t te = tile_elems_for(elem_bytes);
    l.num_tiles = (n + ue - 1) / ue;
    l.num_units1 = (n + te - 1) / te;
    l.num_chunks = (n + (1ull << chunk_log2) - 1) >> chunk_log2;
    // enough statuses for the plain scan (4096 counts per tile); the reduce-then-scan pass
    // keeps its block sums here too (one per 2^18 elements <= one per 64 chunks)
    l.scan_tiles = (l.num_chunks + FUSED_TILE_CHUNKS - 1) / FUSED_TILE_CHUNKS;
    size_t off = sizeof(ws_header);
    l.off_status = off; // one look-back status per unit, for either unit size a column may take
    const uint64_t short_units = l.num_units1 < SHORT_UNITS_MAX ? l.num_units1 : SHORT_UNITS_MAX;
    off += align256(8 * (l.num_tiles > short_units ? l.num_tiles : short_units));
    l.off_scan_status = off;
    off += align256(8 * l.scan_tiles);
    l.off_counts = off;
    off += align256(4 * l.num_chunks);
    l.off_offsets = off;
    off += align256(8 * l.num_chunks);
    l.off_blk_base = off;
    off += align256(8 * ((n + (1ull << SCAN_BLOCK_LOG2) - 1) >> SCAN_BLOCK_LOG2));
    // inside the range the epoch-wrap clear keeps: later kernels of the call read these
    l.off_item_flags = off;
    off += align256(4 * sparse_items_for(n));
    l.off_flags = off;
    off += align256(4 * POPC_FLAG_SLOTS);
    l.total = align256(off);
    return l;
}

struct Resolved {
    int algo;
    uint32_t chunk_log2;
    uint32_t grid;
    uint32_t skip;
    uint64_t timeout_ns;
};

int resolve_config(const cs_config* cfg, uint64_t n, uint32_t elem_bytes, Resolved* r)
{
    cs_config c{};
    if (cfg) c = *cfg;
    uint32_t L = c.chunk_length ? c.chunk_length : 1024u;
    if (!is_pow2(L) || L < 32 || L > 65536) return CS_ERR_INVALID_VALUE;
    if (c.algo < CS_ALGO_AUTO || c.algo > CS_ALGO_NAIVE) return CS_ERR_INVALID_VALUE;
    if (!(c.selectivity >= 0.0f && c.selectivity <= 1.0f)) return CS_ERR_INVALID_VALUE; // NaN too
    r->algo = c.algo;
    r->chunk_log2 = ilog2(L);
    r->grid = c.grid_dim;
    r->skip = (c.skip == 2) ? 0u : 1u;
    r->timeout_ns = c.timeout_ns ? c.timeout_ns : DEFAULT_TIMEOUT_NS;
    if (r->algo == CS_ALGO_AUTO) {
        const TuneChoice t = tune_lookup(n, elem_bytes, c.selectivity);
        r->algo = t.algo;
        if (!(cfg && cfg->chunk_length)) r->chunk_log2 = ilog2(t.chunk_length);
    }
    return CS_SUCCESS;
}

int check_common(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                 uint64_t* d_count)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return CS_ERR_INVALID_VALUE;
    if (!d_count) return CS_ERR_INVALID_VALUE;
    if (n > MAX_N) return CS_ERR_NOT_SUPPORTED;
    if (n == 0) return CS_SUCCESS;
    if (!d_in || !d_mask || !d_out) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_in, elem_bytes) || !aligned(d_out, elem_bytes) || !aligned(d_mask, 4) || !aligned(d_count, 8))
        return CS_ERR_MISALIGNED;
    return CS_SUCCESS;
}

inline int cuda_status(cudaError_t e)
{
    if (e == cudaSuccess) return CS_SUCCESS;
    if (e == cudaErrorMemoryAllocation) return CS_ERR_OUT_OF_MEMORY;
    return CS_ERR_CUDA;
}

uint32_t persistent_grid(uint32_t elem_bytes, int mode, const DeviceInfo& di, uint64_t num_tiles, uint32_t requested,
                         uint32_t unit_tiles = UNIT_TILES)
{
    uint64_t g = requested;
    if (g == 0) {
        int bps = compact_tma_blocks_per_sm(elem_bytes, mode, unit_tiles);
        if (bps < 1) bps = 1;
        g = static_cast<uint64_t>(bps) * di.sms;
    }
    if (g > num_tiles) g = num_tiles;
    if (g == 0) g = 1;
    return static_cast<uint32_t>(g);
}

ColumnDesc make_column(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                       uint64_t* d_count, uint64_t* offsets)
{
    ColumnDesc c{};
    c.in = static_cast<const uint8_t*>(d_in);
    c.mask = static_cast<const uint32_t*>(d_mask);
    c.out = static_cast<uint8_t*>(d_out);
    c.n = n;
    c.d_count = d_count;
    c.offsets = offsets;
    c.elem_bytes = elem_bytes;
    return c;
}

// Pass 3 of the 3-pass form over chunk offsets already in the workspace: independent warps for
// chunk lengths up to 4096 (hybrid: units with at most 1/32 selected are gathered), the
// TMA-staged writeout for longer ones and for skip = 2 (whole tiles are loaded, which warps never do), if
// the pointers allow it.
int launch_writeout_3pass(const ColumnDesc& col, const Layout& l, ws_header* hdr, const Resolved& r, bool hybrid,
                          const uint32_t* item_flags, const DeviceInfo& di, cudaStream_t stream)
{
    const uint32_t elem_bytes = col.elem_bytes;
    const bool whole_tiles = !r.skip && aligned(col.in, 16) && aligned(col.out, 16) && aligned(col.mask, 16);
    if (r.chunk_log2 <= 12 && !whole_tiles) {
        WriteoutParams p{};
        p.col0 = col;
        p.num_units = l.num_tiles;
        p.num_sparse_items = sparse_items_for(col.n);
        p.sparse_max = hybrid ? unit_elems_for(elem_bytes) / 32 : 0;
        p.item_flags = item_flags;
        p.hdr = hdr;
        p.chunk_log2 = r.chunk_log2;
        return cuda_status(launch_writeout_warp(p, elem_bytes, r.grid, di.sms, stream));
    }
    CompactParams p{};
    p.col0 = col;
    p.num_tiles = l.num_tiles;
    p.hdr = hdr;
    p.chunk_log2 = r.chunk_log2;
    p.skip = r.skip;
    p.timeout_ns = r.timeout_ns;
    const uint32_t grid = persistent_grid(elem_bytes, 1, di, l.num_tiles, r.grid);
    return cuda_status(launch_compact_tma(p, elem_bytes, 1, grid, stream));
}

int run_compaction(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                   uint64_t* d_count, void* d_ws, size_t ws_bytes, const Resolved& r, bool auto_route,
                   cudaStream_t stream)
{
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    const Layout l = plan_layout(n, elem_bytes, r.chunk_log2);
    if (!d_ws || ws_bytes < l.total || !aligned(d_ws, 256)) return CS_ERR_WORKSPACE;
    uint8_t* ws = static_cast<uint8_t*>(d_ws);
    ws_header* hdr = reinterpret_cast<ws_header*>(ws);

    int algo = r.algo;
    const bool tma_ok = aligned(d_in, 16) && aligned(d_out, 16) && aligned(d_mask, 16);
    // The 1-pass form runs in slices (cs_slices.cu), or through the TMA kernel for 4- and 8-byte columns of
    // more than slices_per_sm and for skip = 2 (as in launch_writeout_3pass). The slices' totals take the
    // workspace from its look-back statuses on, where a 1-pass call has nothing else: room for 1.19 times as
    // many and more, whatever the chunk length (the least: 2-byte elements, 65536).
    const uint64_t slices = slices_of(n, elem_bytes);
    const bool in_slices =
        r.skip && 8 * slices <= l.total - l.off_status &&
        (elem_bytes <= 2 || slices <= slices_per_sm(elem_bytes) * static_cast<uint64_t>(di.sms));
    if ((algo == CS_ALGO_1PASS || algo == CS_ALGO_3PASS) && !tma_ok) {
        if (!auto_route) return CS_ERR_MISALIGNED;
        // slices take any mask and output, the warp writeout any element-aligned pointers; the latter
        // needs the block pass's offsets
        if (!(algo == CS_ALGO_1PASS && in_slices && aligned(d_in, 16)))
            algo = r.chunk_log2 >= 7 && r.chunk_log2 <= 12 ? CS_ALGO_3PASS : CS_ALGO_NAIVE;
    }

    if (algo == CS_ALGO_1PASS && in_slices) {
        SliceParams p{};
        p.in = static_cast<const uint8_t*>(d_in);
        p.out = static_cast<uint8_t*>(d_out);
        p.mask_in = static_cast<const uint32_t*>(d_mask);
        p.n = n;
        p.d_count = d_count;
        p.hdr = hdr;
        p.status = reinterpret_cast<uint64_t*>(ws + l.off_status);
        p.timeout_ns = r.timeout_ns;
        p.grid = r.grid;
        return cuda_status(launch_onepass(p, elem_bytes, di.sms, stream));
    }
    if (algo == CS_ALGO_1PASS) {
        // a column with fewer full-size units than SMs takes one-tile units, so that about
        // four times as many SMs share it
        const uint32_t unit_tiles =
            l.num_tiles < static_cast<uint64_t>(di.sms) && l.num_units1 <= SHORT_UNITS_MAX ? 1u : UNIT_TILES;
        CompactParams p{};
        p.col0 = make_column(d_in, d_mask, d_out, n, elem_bytes, d_count, nullptr);
        p.num_tiles = unit_tiles == 1u ? l.num_units1 : l.num_tiles;
        p.hdr = hdr;
        p.status = reinterpret_cast<uint64_t*>(ws + l.off_status);
        p.skip = r.skip;
        p.timeout_ns = r.timeout_ns;
        const int mode = (unit_tiles == UNIT_TILES && elem_bytes >= 4 &&
                          l.num_tiles >= DEEP_UNITS_PER_SM * static_cast<uint64_t>(di.sms))
                             ? 2
                             : 0;
        const uint32_t grid = persistent_grid(elem_bytes, mode, di, p.num_tiles, r.grid, unit_tiles);
        return cuda_status(launch_compact_tma(p, elem_bytes, mode, grid, stream, unit_tiles));
    }

    // 3-pass family: popcount -> prefix sum -> writeout
    uint32_t* counts = reinterpret_cast<uint32_t*>(ws + l.off_counts);
    uint64_t* offsets = reinterpret_cast<uint64_t*>(ws + l.off_offsets);
    uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.off_flags);
    const uint64_t ue = unit_elems_for(elem_bytes);
    const bool tma_writeout = algo == CS_ALGO_3PASS && (1ull << r.chunk_log2) <= ue;
    // passes 1 + 2 in one reduce-then-scan launch (block-relative offsets + block prefixes)
    const bool blocks = tma_writeout && r.chunk_log2 >= 7 && r.chunk_log2 <= 12;
    // Only the block pass counts the sparse groups; without it (chunks of 32 and 64) every unit is tested against the
    // share, and the one unit of a short column passes with any selection (4101 u8, 0.95 selected: 3896 elements
    // gathered by one warp, 48 us instead of 15).
    const bool hybrid = algo == CS_ALGO_3PASS && r.chunk_log2 <= 12 && r.skip &&
                        (blocks || sparse_items_for(n) >= GATHER_ITEMS_MIN);
    uint64_t* blk_base = blocks ? reinterpret_cast<uint64_t*>(ws + l.off_blk_base) : nullptr;
    // with the block pass, pass 1 marks the sparse units' items and the gather visits only those
    uint32_t* item_flags = blocks && hybrid ? reinterpret_cast<uint32_t*>(ws + l.off_item_flags) : nullptr;
    cudaError_t e;
    if (blocks) {
        BlockScanParams bp{};
        bp.col0 = make_column(d_in, d_mask, d_out, n, elem_bytes, d_count, offsets);
        bp.col0.blk_base = blk_base;
        bp.num_blocks = (n + (1ull << SCAN_BLOCK_LOG2) - 1) >> SCAN_BLOCK_LOG2;
        bp.blk_sum = reinterpret_cast<uint64_t*>(ws + l.off_scan_status);
        bp.blk_base = blk_base;
        bp.hdr = hdr;
        bp.item_flags = item_flags;
        bp.chunk_log2 = r.chunk_log2;
        bp.keep_begin = l.off_counts;
        bp.keep_end = l.off_flags + 4 * POPC_FLAG_SLOTS;
        e = launch_popc_blocks(bp, di.sms, stream);
        if (e != cudaSuccess) return cuda_status(e);
    } else {
        ScanParams sp{};
        sp.counts = counts;
        sp.count = l.num_chunks;
        sp.offsets = offsets;
        sp.total = d_count;
        sp.hdr = hdr;
        sp.status = reinterpret_cast<uint64_t*>(ws + l.off_scan_status);
        sp.timeout_ns = r.timeout_ns;
        sp.keep_begin = l.off_counts;
        sp.keep_end = l.off_flags + 4 * POPC_FLAG_SLOTS;
        sp.popc_flags = flags;
        e = launch_popc_chunks(static_cast<const uint32_t*>(d_mask), n, r.chunk_log2, counts, hdr, flags, di.sms, stream);
        if (e != cudaSuccess) return cuda_status(e);
        sp.num_tiles = (l.num_chunks + SCAN_TILE - 1) / SCAN_TILE;
        e = launch_scan(sp, di.sms, stream);
        if (e != cudaSuccess) return cuda_status(e);
    }
    ColumnDesc col = make_column(d_in, d_mask, d_out, n, elem_bytes, d_count, offsets);
    col.blk_base = blk_base;
    if (tma_writeout) return launch_writeout_3pass(col, l, hdr, r, hybrid, item_flags, di, stream);
    // chunks longer than a TMA tile, misaligned pointers, or CS_ALGO_NAIVE
    return cuda_status(launch_writeout_naive(d_in, static_cast<const uint32_t*>(d_mask), d_out, n, elem_bytes, offsets,
                                             counts, r.chunk_log2, hdr, di.sms, stream));
}

// ---------------------------------------------------------------------------------
// Library-owned scratch for compressstore / compressstore_cfg / compressstore_if: one
// workspace per (device, stream), grown with stream-ordered allocation so a workspace still
// in use by earlier work on the stream is released only after that work. An entry lives
// until compressstore_release(stream) frees it (a caller that destroys streams calls it
// first; the library cannot tell a destroyed stream's handle from a live one).
// ---------------------------------------------------------------------------------
struct CachedWs {
    void* ptr = nullptr;
    size_t bytes = 0;
};
std::mutex g_ws_mu;
std::map<std::pair<int, cudaStream_t>, CachedWs> g_ws;

int cached_workspace(size_t need, cudaStream_t stream, void** out, size_t* out_bytes)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lk(g_ws_mu);
    CachedWs& c = g_ws[{dev, stream}];
    if (c.bytes < need) {
        size_t want = need < (1u << 20) ? (1u << 20) : need + need / 4;
        want = align256(want);
        void* p = nullptr;
        cudaError_t e = cudaMallocAsync(&p, want, stream);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return CS_ERR_OUT_OF_MEMORY;
        }
        e = launch_ws_init(static_cast<ws_header*>(p), want, stream);
        if (e != cudaSuccess) {
            cudaFreeAsync(p, stream);
            return cuda_status(e);
        }
        if (c.ptr) cudaFreeAsync(c.ptr, stream);
        c.ptr = p;
        c.bytes = want;
    }
    *out = c.ptr;
    *out_bytes = c.bytes;
    return CS_SUCCESS;
}

// Free the cached workspace of (current device, stream), in the stream's order.
int release_cached_workspace(cudaStream_t stream)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lk(g_ws_mu);
    auto it = g_ws.find({dev, stream});
    if (it == g_ws.end()) return CS_SUCCESS;
    const cudaError_t e = it->second.ptr ? cudaFreeAsync(it->second.ptr, stream) : cudaSuccess;
    g_ws.erase(it);
    return cuda_status(e);
}

int lookup_cached_workspace(cudaStream_t stream, void** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CS_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lk(g_ws_mu);
    auto it = g_ws.find({dev, stream});
    if (it == g_ws.end()) {
        *out = nullptr;
        return CS_SUCCESS;
    }
    *out = it->second.ptr;
    return CS_SUCCESS;
}

int check_workspace_error(void* d_ws, cudaStream_t stream)
{
    cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_status(e);
    if (!d_ws) return CS_SUCCESS;
    uint32_t err = 0;
    ws_header* hdr = static_cast<ws_header*>(d_ws);
    e = cudaMemcpy(&err, &hdr->err, sizeof(err), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_status(e);
    if (err == 0) return CS_SUCCESS;
    e = cudaMemset(&hdr->err, 0, sizeof(uint32_t));
    if (e != cudaSuccess) return cuda_status(e);
    return err == DEVERR_RANGE ? CS_ERR_INVALID_VALUE : CS_ERR_TIMEOUT;
}

// The predicate as lo <= x <= hi, negated for NE (and for a selection of nothing): inclusive bounds
// of whole numbers, hi as the distance from lo; of floating numbers the neighbouring values.
template <typename T>
void predicate_bounds_t(const cs_predicate& pr, SliceParams& p)
{
    constexpr bool REAL = std::numeric_limits<T>::has_infinity;
    T a, b;
    std::memcpy(&a, &pr.a, sizeof(T));
    std::memcpy(&b, &pr.b, sizeof(T));
    const T lowest = REAL ? -std::numeric_limits<T>::infinity() : std::numeric_limits<T>::lowest();
    const T highest = REAL ? std::numeric_limits<T>::infinity() : std::numeric_limits<T>::max();
    T lo = lowest, hi = highest;
    bool none = false, neg = false;
    // the largest value below a, the smallest above it
    auto below = [&]() -> T {
        if constexpr (REAL) return std::nextafter(a, lowest);
        else return static_cast<T>(a - 1);
    };
    auto above = [&]() -> T {
        if constexpr (REAL) return std::nextafter(a, highest);
        else return static_cast<T>(a + 1);
    };
    switch (pr.op) {
        case CS_PRED_LT:
            none = !(a > lowest); // a NaN too
            if (!none) hi = below();
            break;
        case CS_PRED_LE: hi = a; break; // a NaN compares false
        case CS_PRED_GT:
            none = !(a < highest);
            if (!none) lo = above();
            break;
        case CS_PRED_GE: lo = a; break;
        case CS_PRED_EQ: lo = hi = a; break;
        case CS_PRED_NE: lo = hi = a; neg = true; break;
        default: // CS_PRED_BETWEEN
            lo = a;
            hi = b;
            none = !(lo <= hi);
            break;
    }
    if constexpr (REAL) {
        if (none) lo = highest, hi = lowest;
    } else {
        if (none) lo = lowest, hi = highest, neg = true;
        using U = typename std::make_unsigned<T>::type;
        const U rng = static_cast<U>(static_cast<U>(hi) - static_cast<U>(lo));
        std::memcpy(&hi, &rng, sizeof(T));
    }
    p.lo = p.hi = 0;
    std::memcpy(&p.lo, &lo, sizeof(T));
    std::memcpy(&p.hi, &hi, sizeof(T));
    p.negate = neg;
    p.sides = none ? 3u : pr.op == CS_PRED_GT || pr.op == CS_PRED_GE ? 1u : pr.op == CS_PRED_LT || pr.op == CS_PRED_LE ? 2u : 3u;
}

// Element width of a cs_elem_type and its bounds; 0 for an unknown type.
uint32_t predicate_bounds(const cs_predicate& pr, SliceParams& p)
{
    switch (pr.type) {
        case CS_U8: predicate_bounds_t<uint8_t>(pr, p); return 1;
        case CS_U16: predicate_bounds_t<uint16_t>(pr, p); return 2;
        case CS_U32: predicate_bounds_t<uint32_t>(pr, p); return 4;
        case CS_U64: predicate_bounds_t<uint64_t>(pr, p); return 8;
        case CS_I8: predicate_bounds_t<int8_t>(pr, p); return 1;
        case CS_I16: predicate_bounds_t<int16_t>(pr, p); return 2;
        case CS_I32: predicate_bounds_t<int32_t>(pr, p); return 4;
        case CS_I64: predicate_bounds_t<int64_t>(pr, p); return 8;
        case CS_F32: predicate_bounds_t<float>(pr, p); return 4;
        case CS_F64: predicate_bounds_t<double>(pr, p); return 8;
        default: return 0;
    }
}

} // namespace
} // namespace cs

using namespace cs;

extern "C" {

size_t compressstore_workspace_size(uint64_t n, uint32_t elem_bytes, const cs_config* cfg)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return 0;
    Resolved r{};
    if (resolve_config(cfg, n, elem_bytes, &r) != CS_SUCCESS) return 0;
    return plan_layout(n, elem_bytes, r.chunk_log2).total;
}

int cs_workspace_init(void* d_ws, size_t ws_bytes, cs_stream_t stream)
{
    if (!d_ws || ws_bytes < sizeof(ws_header) || !aligned(d_ws, 256)) return CS_ERR_WORKSPACE;
    return cuda_status(launch_ws_init(static_cast<ws_header*>(d_ws), ws_bytes & ~static_cast<size_t>(15),
                                      reinterpret_cast<cudaStream_t>(stream)));
}

int compressstore_ex(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                     uint64_t* d_count, void* d_ws, size_t ws_bytes, const cs_config* cfg, cs_stream_t stream)
{
    int st = check_common(d_in, d_mask, d_out, n, elem_bytes, d_count);
    if (st) return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) return cuda_status(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
    Resolved r{};
    st = resolve_config(cfg, n, elem_bytes, &r);
    if (st) return st;
    const bool auto_route = !(cfg && cfg->algo != CS_ALGO_AUTO);
    return run_compaction(d_in, d_mask, d_out, n, elem_bytes, d_count, d_ws, ws_bytes, r, auto_route, s);
}

int compressstore_cfg(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                      uint64_t* d_count, const cs_config* cfg, cs_stream_t stream)
{
    int st = check_common(d_in, d_mask, d_out, n, elem_bytes, d_count);
    if (st) return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) return cuda_status(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
    DeviceInfo di;
    st = current_device_info(&di);
    if (st) return st;
    Resolved r{};
    st = resolve_config(cfg, n, elem_bytes, &r);
    if (st) return st;
    const size_t need = plan_layout(n, elem_bytes, r.chunk_log2).total;
    void* ws = nullptr;
    size_t ws_bytes = 0;
    st = cached_workspace(need, s, &ws, &ws_bytes);
    if (st) return st;
    const bool auto_route = !(cfg && cfg->algo != CS_ALGO_AUTO);
    return run_compaction(d_in, d_mask, d_out, n, elem_bytes, d_count, ws, ws_bytes, r, auto_route, s);
}

int compressstore(const void* d_in, const void* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                  uint64_t* d_count, cs_stream_t stream)
{
    return compressstore_cfg(d_in, d_mask, d_out, n, elem_bytes, d_count, nullptr, stream);
}

int compressstore_if(const void* d_in, void* d_out, uint64_t n, const cs_predicate* pred, uint32_t* d_mask_out,
                     uint64_t* d_count, cs_stream_t stream)
{
    if (!pred || !d_count) return CS_ERR_INVALID_VALUE;
    if (pred->op < CS_PRED_LT || pred->op > CS_PRED_BETWEEN) return CS_ERR_INVALID_VALUE;
    SliceParams p{};
    const uint32_t w = predicate_bounds(*pred, p);
    if (w == 0) return CS_ERR_INVALID_VALUE;
    if (n > MAX_N) return CS_ERR_NOT_SUPPORTED;
    if (!aligned(d_count, 8)) return CS_ERR_MISALIGNED;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n == 0) return cuda_status(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
    if (!d_in || !d_out) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_in, 16) || !aligned(d_out, 16) || (d_mask_out && !aligned(d_mask_out, 16))) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    const size_t need = align256(sizeof(ws_header) + 8 * slices_of(n, w));
    void* ws = nullptr;
    size_t ws_bytes = 0;
    st = cached_workspace(need, s, &ws, &ws_bytes);
    if (st) return st;
    p.in = static_cast<const uint8_t*>(d_in);
    p.out = static_cast<uint8_t*>(d_out);
    p.mask = d_mask_out;
    p.n = n;
    p.d_count = d_count;
    p.hdr = static_cast<ws_header*>(ws);
    p.status = reinterpret_cast<uint64_t*>(static_cast<uint8_t*>(ws) + sizeof(ws_header));
    p.timeout_ns = DEFAULT_TIMEOUT_NS;
    return cuda_status(launch_if(p, pred->type, di.sms, s));
}

int cs_workspace_check(void* d_ws, cs_stream_t stream)
{
    return check_workspace_error(d_ws, reinterpret_cast<cudaStream_t>(stream));
}

int compressstore_release(cs_stream_t stream)
{
    return release_cached_workspace(reinterpret_cast<cudaStream_t>(stream));
}

int compressstore_check(cs_stream_t stream)
{
    void* ws = nullptr;
    int st = lookup_cached_workspace(reinterpret_cast<cudaStream_t>(stream), &ws);
    if (st) return st;
    return check_workspace_error(ws, reinterpret_cast<cudaStream_t>(stream));
}

int cs_popc_chunks(const uint32_t* d_mask, uint64_t n, uint32_t chunk_length, uint32_t* d_chunk_counts,
                   cs_stream_t stream)
{
    if (!is_pow2(chunk_length) || chunk_length < 32 || chunk_length > 65536) return CS_ERR_INVALID_VALUE;
    if (n > MAX_N) return CS_ERR_NOT_SUPPORTED;
    if (n == 0) return CS_SUCCESS;
    if (!d_mask || !d_chunk_counts) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_mask, 4) || !aligned(d_chunk_counts, 4)) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    return cuda_status(launch_popc_chunks(d_mask, n, ilog2(chunk_length), d_chunk_counts, nullptr, nullptr, di.sms,
                                          reinterpret_cast<cudaStream_t>(stream)));
}

size_t cs_scan_workspace_size(uint64_t chunk_count)
{
    const uint64_t tiles = (chunk_count + SCAN_TILE - 1) / SCAN_TILE;
    return align256(sizeof(ws_header) + align256(8 * tiles));
}

int cs_chunk_prefix_sum(const uint32_t* d_chunk_counts, uint64_t chunk_count, uint64_t* d_chunk_offsets,
                        uint64_t* d_total, void* d_ws, size_t ws_bytes, cs_stream_t stream)
{
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (chunk_count == 0) {
        if (d_total) return cuda_status(cudaMemsetAsync(d_total, 0, sizeof(uint64_t), s));
        return CS_SUCCESS;
    }
    if (!d_chunk_counts || !d_chunk_offsets) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_chunk_counts, 4) || !aligned(d_chunk_offsets, 8) || (d_total && !aligned(d_total, 8)))
        return CS_ERR_MISALIGNED;
    if (!d_ws || ws_bytes < cs_scan_workspace_size(chunk_count) || !aligned(d_ws, 256)) return CS_ERR_WORKSPACE;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    uint8_t* ws = static_cast<uint8_t*>(d_ws);
    ScanParams sp{};
    sp.counts = d_chunk_counts;
    sp.count = chunk_count;
    sp.offsets = d_chunk_offsets;
    sp.total = d_total;
    sp.hdr = reinterpret_cast<ws_header*>(ws);
    sp.status = reinterpret_cast<uint64_t*>(ws + sizeof(ws_header));
    sp.num_tiles = (chunk_count + SCAN_TILE - 1) / SCAN_TILE;
    sp.timeout_ns = DEFAULT_TIMEOUT_NS;
    return cuda_status(launch_scan(sp, di.sms, s));
}

int cs_writeout(const void* d_in, const uint32_t* d_mask, void* d_out, uint64_t n, uint32_t elem_bytes,
                const uint64_t* d_chunk_offsets, const uint32_t* d_chunk_counts, uint32_t chunk_length, int32_t algo,
                cs_stream_t stream)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return CS_ERR_INVALID_VALUE;
    if (!is_pow2(chunk_length) || chunk_length < 32 || chunk_length > 65536) return CS_ERR_INVALID_VALUE;
    if (algo != CS_ALGO_3PASS && algo != CS_ALGO_NAIVE) return CS_ERR_INVALID_VALUE;
    if (n > MAX_N) return CS_ERR_NOT_SUPPORTED;
    if (n == 0) return CS_SUCCESS;
    if (!d_in || !d_mask || !d_out || !d_chunk_offsets) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_in, elem_bytes) || !aligned(d_out, elem_bytes) || !aligned(d_mask, 4) ||
        !aligned(d_chunk_offsets, 8))
        return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t log2L = ilog2(chunk_length);
    const uint64_t ue = unit_elems_for(elem_bytes);
    if (algo == CS_ALGO_3PASS) {
        if (!(aligned(d_in, 16) && aligned(d_out, 16) && aligned(d_mask, 16))) return CS_ERR_MISALIGNED;
        if (chunk_length > ue) return CS_ERR_NOT_SUPPORTED;
        // no workspace: errors are not recorded, inconsistent offsets still never write
        const ColumnDesc col =
            make_column(d_in, d_mask, d_out, n, elem_bytes, nullptr, const_cast<uint64_t*>(d_chunk_offsets));
        if (log2L <= 12) {
            WriteoutParams p{};
            p.col0 = col;
            p.num_units = (n + ue - 1) / ue;
            p.chunk_log2 = log2L;
            return cuda_status(launch_writeout_warp(p, elem_bytes, 0, di.sms, s));
        }
        CompactParams p{};
        p.col0 = col;
        p.num_tiles = (n + ue - 1) / ue;
        p.chunk_log2 = log2L;
        p.skip = 1;
        p.timeout_ns = DEFAULT_TIMEOUT_NS;
        const uint32_t grid = persistent_grid(elem_bytes, 1, di, p.num_tiles, 0);
        return cuda_status(launch_compact_tma(p, elem_bytes, 1, grid, s));
    }
    return cuda_status(launch_writeout_naive(d_in, d_mask, d_out, n, elem_bytes, d_chunk_offsets, d_chunk_counts, log2L,
                                             nullptr, di.sms, s));
}

int cs_gen_payload(void* d_out, uint64_t n, uint32_t elem_bytes, uint64_t seed, int32_t float_unit, cs_stream_t stream)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return CS_ERR_INVALID_VALUE;
    if (n == 0) return CS_SUCCESS;
    if (!d_out) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_out, elem_bytes)) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    return cuda_status(
        launch_gen_payload(d_out, n, elem_bytes, seed, float_unit, di.sms, reinterpret_cast<cudaStream_t>(stream)));
}

int cs_gen_mask_bernoulli(uint32_t* d_mask, uint64_t n, double p, uint64_t seed, cs_stream_t stream)
{
    if (n == 0) return CS_SUCCESS;
    if (!d_mask || !(p >= 0.0 && p <= 1.0)) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_mask, 4)) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    const uint64_t thr = (p >= 1.0) ? (1ull << 32) : static_cast<uint64_t>(p * 4294967296.0);
    return cuda_status(launch_gen_mask_bernoulli(d_mask, n, thr, seed, di.sms, reinterpret_cast<cudaStream_t>(stream)));
}

size_t cs_gen_mask_runs_workspace_size(uint64_t n)
{
    const uint64_t nw = (n + 31) / 32;
    return cs_scan_workspace_size(nw) + align256(4 * nw) + align256(8 * nw);
}

int cs_gen_mask_runs(uint32_t* d_mask, uint64_t n, double mean_run, uint64_t seed, void* d_ws, size_t ws_bytes,
                     cs_stream_t stream)
{
    if (n == 0) return CS_SUCCESS;
    if (!d_mask || !(mean_run >= 1.0)) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_mask, 4)) return CS_ERR_MISALIGNED;
    if (!d_ws || ws_bytes < cs_gen_mask_runs_workspace_size(n) || !aligned(d_ws, 256)) return CS_ERR_WORKSPACE;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const uint64_t nw = (n + 31) / 32;
    const uint64_t thr = static_cast<uint64_t>(4294967296.0 / mean_run);
    uint8_t* ws = static_cast<uint8_t*>(d_ws);
    const size_t scan_bytes = cs_scan_workspace_size(nw);
    uint32_t* counts = reinterpret_cast<uint32_t*>(ws + scan_bytes);
    uint64_t* offsets = reinterpret_cast<uint64_t*>(ws + scan_bytes + align256(4 * nw));
    cudaError_t e = launch_gen_runs_toggle(d_mask, counts, n, thr, seed, di.sms, s);
    if (e != cudaSuccess) return cuda_status(e);
    ScanParams sp{};
    sp.counts = counts;
    sp.count = nw;
    sp.offsets = offsets;
    sp.total = nullptr;
    sp.hdr = reinterpret_cast<ws_header*>(ws);
    sp.status = reinterpret_cast<uint64_t*>(ws + sizeof(ws_header));
    sp.num_tiles = (nw + SCAN_TILE - 1) / SCAN_TILE;
    sp.timeout_ns = DEFAULT_TIMEOUT_NS;
    sp.keep_begin = scan_bytes;
    sp.keep_end = scan_bytes + align256(4 * nw) + 8 * nw;
    e = launch_scan(sp, di.sms, s);
    if (e != cudaSuccess) return cuda_status(e);
    return cuda_status(launch_gen_runs_apply(d_mask, offsets, n, di.sms, s));
}

int cs_gen_mask_dense_prefix(uint32_t* d_mask, uint64_t n, float frac, cs_stream_t stream)
{
    if (n == 0) return CS_SUCCESS;
    if (!d_mask || !(frac >= 0.0f)) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_mask, 4)) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    uint64_t k = static_cast<uint64_t>(frac * static_cast<float>(n));
    if (k > n) k = n;
    return cuda_status(launch_gen_mask_dense_prefix(d_mask, n, k, di.sms, reinterpret_cast<cudaStream_t>(stream)));
}

int cs_gen_mask_pattern(uint32_t* d_mask, uint64_t n, uint32_t pattern, uint32_t pattern_length, cs_stream_t stream)
{
    if (pattern_length < 1 || pattern_length > 32) return CS_ERR_INVALID_VALUE;
    if (n == 0) return CS_SUCCESS;
    if (!d_mask) return CS_ERR_INVALID_VALUE;
    if (!aligned(d_mask, 4)) return CS_ERR_MISALIGNED;
    DeviceInfo di;
    int st = current_device_info(&di);
    if (st) return st;
    const uint32_t pm = pattern_length >= 32 ? pattern : (pattern & ((1u << pattern_length) - 1u));
    return cuda_status(
        launch_gen_mask_pattern(d_mask, n, pm, pattern_length, di.sms, reinterpret_cast<cudaStream_t>(stream)));
}

const char* cs_status_string(int status)
{
    switch (status) {
        case CS_PENDING: return "pending";
        case CS_SUCCESS: return "success";
        case CS_ERR_INVALID_VALUE: return "invalid value";
        case CS_ERR_MISALIGNED: return "misaligned pointer";
        case CS_ERR_WORKSPACE: return "workspace missing, too small or misaligned";
        case CS_ERR_CUDA: return "CUDA runtime error";
        case CS_ERR_TIMEOUT: return "bounded device wait timed out";
        case CS_ERR_NO_DEVICE: return "no usable sm_100 device";
        case CS_ERR_OUT_OF_MEMORY: return "out of device memory";
        case CS_ERR_NOT_SUPPORTED: return "not supported";
        case CS_ERR_ADMISSION: return "request exceeds the memory budget";
        default: return "unknown status";
    }
}

uint64_t cs_launch_count(void)
{
    return g_launches.load(std::memory_order_relaxed);
}

uint32_t cs_tile_elems(uint32_t elem_bytes)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return 0;
    return tile_elems_for(elem_bytes);
}

uint32_t cs_compact_smem_bytes(uint32_t elem_bytes, int32_t algo)
{
    if (algo != CS_ALGO_1PASS && algo != CS_ALGO_3PASS) return 0;
    if (algo == CS_ALGO_3PASS) return compact_tma_smem_bytes(elem_bytes, 1);
    const uint32_t a = compact_tma_smem_bytes(elem_bytes, 0), b = compact_tma_smem_bytes(elem_bytes, 2);
    return a > b ? a : b; // the largest a 1-pass call may launch
}

uint32_t cs_version(void)
{
    return 0x000100u;
}

} // extern "C"
