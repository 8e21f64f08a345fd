// cs_kernels.cu — chunk popcount (pass 1), single-pass look-back scan (pass 2),
// warp-per-word writeout (the alignment-agnostic pass 3), workspace init and the seeded
// input generators.
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "cs_internal.cuh"

namespace cs {

// ---------------------------------------------------------------------------------
// Pass 1: per-chunk popcount.
// Reference: kernel_3pass_popc_none_striding (src/kernels/kernel_3pass.cuh:12-38) assigns
// one thread per chunk and walks it with strided 4-byte loads. Here consecutive threads
// read consecutive mask words (fully coalesced) and chunks are reduced with shuffles:
// chunks of <= 32 words are segmented warp reductions, longer chunks are warp-strided.
// Bits at positions >= n are masked off, so the mask tail need not be zero.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t load_mask_word(const uint32_t* mask, uint64_t wi, uint64_t nw, uint64_t n)
{
    if (wi >= nw) return 0u;
    uint32_t m = __ldg(mask + wi);
    if (wi == nw - 1 && (n & 31u)) m &= (1u << (n & 31u)) - 1u;
    return m;
}

// Vector form (16-byte-aligned mask, 128 <= L <= 4096): a warp step reads 32 uint4 (128 words
// = 4096 elements) and four steps are unrolled so four loads per lane are in flight; chunks
// of LPC = L/128 lanes are reduced with xor shuffles. Each unrolled warp iteration covers an
// aligned block of 16384 elements; when `hdr` is given, each CTA records in cta_flags whether
// one of its blocks holds at most 16384/32 selected elements, and the scan that follows
// turns that into hdr->sparse_epoch so the hybrid writeout knows to look for sparse units.
template <int LPC>
__global__ void __launch_bounds__(256) k_popc_chunks_vec(const uint32_t* __restrict__ mask, uint64_t n,
                                                         uint32_t* __restrict__ counts, ws_header* hdr,
                                                         uint32_t* __restrict__ cta_flags)
{
    __shared__ uint32_t s_sparse;
    if (threadIdx.x == 0) s_sparse = 0;
    __syncthreads();
    constexpr int UNROLL = 4;
    const uint64_t nw = (n + 31) / 32;
    const uint64_t nvec = (nw + 3) / 4;
    const uint64_t num_chunks = (nw + 4 * LPC - 1) / (4 * LPC);
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp_global = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t total_warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    const uint4* mv = reinterpret_cast<const uint4*>(mask);
    bool sparse_block = false;
    for (uint64_t base = warp_global * 32 * UNROLL; base < nvec; base += total_warps * 32 * UNROLL) {
        uint4 q[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const uint64_t v = base + u * 32 + lane;
            if (v * 4 + 3 < nw) {
                q[u] = __ldg(mv + v);
                if (v * 4 + 3 == nw - 1 && (n & 31u)) q[u].w &= (1u << (n & 31u)) - 1u;
            } else {
                q[u].x = load_mask_word(mask, v * 4 + 0, nw, n);
                q[u].y = load_mask_word(mask, v * 4 + 1, nw, n);
                q[u].z = load_mask_word(mask, v * 4 + 2, nw, n);
                q[u].w = load_mask_word(mask, v * 4 + 3, nw, n);
            }
        }
        uint32_t block = 0;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            uint32_t c = __popc(q[u].x) + __popc(q[u].y) + __popc(q[u].z) + __popc(q[u].w);
            block += c;
#pragma unroll
            for (int d = LPC / 2; d > 0; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
            const uint64_t chunk = (base + u * 32 + lane) / LPC;
            if ((lane % LPC) == 0 && chunk < num_chunks) counts[chunk] = c;
        }
        if (hdr) {
            block = warp_sum32(block);
            sparse_block |= block <= (16384u / 32u);
        }
    }
    // one flag word per CTA (distinct addresses: same-address stores from every warp would
    // serialise in L2); the scan's last CTA folds them into hdr->sparse_epoch
    if (hdr) {
        if (lane == 0 && sparse_block) s_sparse = 1u;
        __syncthreads();
        if (threadIdx.x == 0) {
            if (blockIdx.x == 0) hdr->popc_ctas = gridDim.x;
            cta_flags[blockIdx.x] = s_sparse ? epoch_mark(hdr->epoch) : 0u;
        }
    }
}

// Scalar form (any 4-byte-aligned mask, any chunk length). It never proves the absence of
// sparse blocks, so with `hdr` it always flags the call.
__global__ void __launch_bounds__(256) k_popc_chunks(const uint32_t* __restrict__ mask, uint64_t n, uint32_t chunk_log2,
                                                     uint32_t* __restrict__ counts, ws_header* hdr,
                                                     uint32_t* __restrict__ cta_flags)
{
    const uint64_t nw = (n + 31) / 32;
    const uint32_t wpc_log2 = chunk_log2 - 5; // words per chunk = 2^wpc_log2
    const uint64_t num_chunks = (n + (1ull << chunk_log2) - 1) >> chunk_log2;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp_global = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t total_warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    if (hdr && blockIdx.x == 0 && threadIdx.x == 0) {
        hdr->popc_ctas = 1;
        cta_flags[0] = epoch_mark(hdr->epoch);
    }
    if (wpc_log2 <= 5) {
        const uint32_t wpc = 1u << wpc_log2;
        const uint64_t nw_round = (nw + 31) & ~31ull;
        for (uint64_t base = warp_global * 32; base < nw_round; base += total_warps * 32) {
            const uint64_t wi = base + lane;
            uint32_t c = __popc(load_mask_word(mask, wi, nw, n));
            for (uint32_t off = wpc >> 1; off > 0; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
            if ((lane & (wpc - 1)) == 0) {
                const uint64_t chunk = wi >> wpc_log2;
                if (chunk < num_chunks) counts[chunk] = c;
            }
        }
    } else {
        const uint64_t wpc = 1ull << wpc_log2;
        for (uint64_t chunk = warp_global; chunk < num_chunks; chunk += total_warps) {
            uint32_t c = 0;
            const uint64_t w0 = chunk * wpc;
            for (uint64_t wi = w0 + lane; wi < w0 + wpc; wi += 32) c += __popc(load_mask_word(mask, wi, nw, n));
            c = warp_sum32(c);
            if (lane == 0) counts[chunk] = c;
        }
    }
}

cudaError_t launch_popc_chunks(const uint32_t* mask, uint64_t n, uint32_t chunk_log2, uint32_t* counts, ws_header* hdr,
                               uint32_t* cta_flags, int num_sms, cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    const bool vec = (reinterpret_cast<uintptr_t>(mask) & 15u) == 0 && chunk_log2 >= 7 && chunk_log2 <= 12;
    if (vec) {
        uint64_t blocks = ((nw + 3) / 4 + 1023) / 1024; // 8 warps x 128 vectors per block iteration
        uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
        if (cap > POPC_FLAG_SLOTS) cap = POPC_FLAG_SLOTS;
        if (blocks > cap) blocks = cap;
        if (blocks == 0) blocks = 1;
        const unsigned g = static_cast<unsigned>(blocks);
        switch (chunk_log2) {
            case 7: k_popc_chunks_vec<1><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
            case 8: k_popc_chunks_vec<2><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
            case 9: k_popc_chunks_vec<4><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
            case 10: k_popc_chunks_vec<8><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
            case 11: k_popc_chunks_vec<16><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
            default: k_popc_chunks_vec<32><<<g, 256, 0, stream>>>(mask, n, counts, hdr, cta_flags); break;
        }
    } else {
        uint64_t blocks = (nw + 255) / 256;
        const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
        if (blocks > cap) blocks = cap;
        if (blocks == 0) blocks = 1;
        k_popc_chunks<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, n, chunk_log2, counts, hdr,
                                                                          cta_flags);
    }
    note_launch();
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Pass 2: exclusive prefix sum of chunk counts, single pass with decoupled look-back.
// Reference: the hand-written up-sweep tree (kernel_3pass_pss_gmem_*, log2(C) launches,
// src/kernels/kernel_3pass.cuh:69-153) plus d_3pass_pproc_pssidx (:155-185), and the CUB
// ExclusiveSum it was replaced by (src/cub_wraps.cuh:52-79). Tiles of 4096 counts are
// taken in order from a device counter, so a tile only ever waits on tiles already held
// by running CTAs. The last tile writes the grand total (the selected count).
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(ScanParams p)
{
    __shared__ uint64_t s_warp[SCAN_THREADS / 32];
    __shared__ uint64_t s_tile_total;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_flag;
    __shared__ LookbackSmem<SCAN_THREADS / 32> s_lb;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint32_t epoch = p.hdr->epoch;

    while (true) {
        if (tid == 0) s_tile = atomicAdd(&p.hdr->scan_tile_counter, 1u);
        __syncthreads();
        const uint64_t tile = s_tile;
        if (tile >= p.num_tiles) break;
        const uint64_t base = tile * SCAN_TILE + static_cast<uint64_t>(tid) * SCAN_ITEMS_PER_THREAD;
        uint32_t v[SCAN_ITEMS_PER_THREAD];
        if (base + SCAN_ITEMS_PER_THREAD <= p.count && (reinterpret_cast<uintptr_t>(p.counts) & 15u) == 0) {
            const uint4* q = reinterpret_cast<const uint4*>(p.counts + base);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 x = __ldg(q + i);
                v[4 * i + 0] = x.x;
                v[4 * i + 1] = x.y;
                v[4 * i + 2] = x.z;
                v[4 * i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < (int)SCAN_ITEMS_PER_THREAD; ++i) v[i] = (base + i < p.count) ? __ldg(p.counts + base + i) : 0u;
        }
        uint64_t thread_total = 0;
#pragma unroll
        for (int i = 0; i < (int)SCAN_ITEMS_PER_THREAD; ++i) thread_total += v[i];
        const uint64_t incl = warp_incl_scan64(thread_total, lane);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint64_t wt = lane < SCAN_THREADS / 32 ? s_warp[lane] : 0ull;
            const uint64_t wincl = warp_incl_scan64(wt, lane);
            const uint64_t tile_total = __shfl_sync(0xffffffffu, wincl, SCAN_THREADS / 32 - 1);
            if (lane < SCAN_THREADS / 32) s_warp[lane] = wincl - wt;
            if (lane == 0) s_tile_total = tile_total;
        }
        __syncthreads();
        const uint64_t prefix =
            lookback_cta<SCAN_THREADS>(p.status, tile, s_tile_total, epoch, p.timeout_ns, p.hdr, s_lb);
        if (prefix == POISON) {
#pragma unroll
            for (int i = 0; i < (int)SCAN_ITEMS_PER_THREAD; ++i)
                if (base + i < p.count) p.offsets[base + i] = POISON;
            if (tile == p.num_tiles - 1 && tid == 0 && p.total) *p.total = POISON;
        } else {
            uint64_t run = prefix + s_warp[warp] + (incl - thread_total);
#pragma unroll
            for (int i = 0; i < (int)SCAN_ITEMS_PER_THREAD; ++i) {
                if (base + i < p.count) p.offsets[base + i] = run;
                run += v[i];
            }
            if (tile == p.num_tiles - 1 && tid == 0 && p.total) *p.total = prefix + s_tile_total;
        }
        __syncthreads();
    }
    lookback_kernel_epilogue(p.hdr, &p.hdr->scan_tile_counter, &p.hdr->scan_done_counter, &s_flag, true, p.keep_begin,
                             p.keep_end, p.popc_flags);
}

cudaError_t launch_scan(const ScanParams& p, int num_sms, cudaStream_t stream)
{
    uint64_t blocks = p.num_tiles;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 4;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_scan<<<static_cast<unsigned>(blocks), SCAN_THREADS, 0, stream>>>(p);
    note_launch();
    return cudaGetLastError();
}


// Pass 1 of the hybrid writeout: the units of block `bl` of a column (UE = 131072 / w
// elements = 32 / w rows of 4096, always whole inside a 2^18-element block) whose count is
// at most UE / 32 belong to the sparse gather: their 16K-element items get this call's
// epoch_mark in p.item_flags, and the gather visits only items so marked (an earlier call's mark that
// is the same costs the gather one test of the offsets, never a wrong write).
// s_warp / s_whalf: selected elements in each warp's 8 rows and in their first 4 rows.
// Called by all threads after those are written.
template <typename Col>
__device__ __forceinline__ void mark_sparse_units(const BlockScanParams& p, const Col& col, uint64_t bl,
                                                  const uint32_t* s_warp, const uint32_t* s_whalf, uint32_t epoch)
{
    const uint32_t w = col.elem_bytes;
    const uint32_t rpu = 32u / w;     // rows per unit
    const uint32_t units = 64u / rpu; // units per block
    const uint32_t t = threadIdx.x;
    if (t >= units) return;
    uint32_t cnt;
    if (w == 8) cnt = (t & 1u) ? s_warp[t >> 1] - s_whalf[t >> 1] : s_whalf[t >> 1];
    else if (w == 4) cnt = s_warp[t];
    else if (w == 2) cnt = s_warp[2 * t] + s_warp[2 * t + 1];
    else cnt = s_warp[4 * t] + s_warp[4 * t + 1] + s_warp[4 * t + 2] + s_warp[4 * t + 3];
    const uint64_t ue = 131072u / w;
    const uint64_t e0 = (bl << SCAN_BLOCK_LOG2) + static_cast<uint64_t>(t) * ue;
    if (e0 >= col.n || cnt > ue / 32) return;
    const uint64_t e1 = e0 + ue < col.n ? e0 + ue : col.n;
    const uint32_t mark = epoch_mark(epoch);
    for (uint64_t it = e0 / 16384; it < (e1 + 16383) / 16384; ++it) p.item_flags[col.item_base + it] = mark;
}

// ---------------------------------------------------------------------------------
// Pass 1 + 2 as one reduce-then-scan kernel (3-pass form, chunk length L = 128 .. 4096). A column is cut into blocks of 2^18 elements (32 KB of mask). A
// CTA takes whole blocks by static assignment and never waits on another CTA: its 8 warps
// each load 8 rows of 32 uint4 (4096 elements per row) in one round, each lane's share of a
// chunk is summed over the LPC = L/128 lanes holding the chunk, and warp and block scans
// give every chunk its offset within the block; the block's sum goes to blk_sum. The last
// CTA to finish scans the block sums into blk_base (exclusive prefix of each block within
// its column) and writes every column's count; consumers add the two (chunk_offset). This
// replaces a decoupled look-back across blocks, whose waiting dominated the fused pass at
// large n. Each CTA also counts its whole 16K-element groups of at most 512 selected
// elements (the hint by which the writeout takes its gather, SPARSE_GROUPS_MIN).
// Reference: pass 1 kernel_3pass_popc_none_striding (src/kernels/kernel_3pass.cuh:12-57)
// and pass 2 launch_cub_pss / kernel_3pass_pss_gmem (src/cub_wraps.cuh:52-79,
// src/kernels/kernel_3pass.cuh:59-214).
// ---------------------------------------------------------------------------------

// A block's share of its column's mask: `words` words, of which the first 4 * groups are whole
// 16-byte groups that can be read as such (none where the mask starts inside a group).
struct PopcShare {
    uint32_t words;
    uint32_t groups;
    uint32_t last_bits; // bits of the last word, 0 if all 32
};

template <typename Col>
__device__ __forceinline__ PopcShare popc_share(const Col& col, uint64_t bl)
{
    const uint64_t left = col.n - (bl << SCAN_BLOCK_LOG2);
    if (left >= (1ull << SCAN_BLOCK_LOG2)) {
        constexpr uint32_t WORDS = (1u << SCAN_BLOCK_LOG2) / 32;
        return {WORDS, (reinterpret_cast<uintptr_t>(col.mask) & 15u) == 0 ? WORDS / 4 : 0u, 0u};
    }
    const uint32_t l = static_cast<uint32_t>(left);
    const uint32_t words = (l + 31u) / 32u;
    return {words, (reinterpret_cast<uintptr_t>(col.mask) & 15u) == 0 ? words / 4u : 0u, l & 31u};
}

// The end of a column's mask, once its whole groups are in q and the rest of q is 0: the words past
// the last whole group are read one by one, and the bits past the column's end cleared.
__device__ __forceinline__ void popc_mask_end(const uint32_t* words, const PopcShare& sh, uint32_t warp, uint32_t lane,
                                              uint4 (&q)[8])
{
    const uint32_t g = (sh.words - 1u) / 4u; // the group with the last word
    if (g / 256u != warp || (g & 31u) != lane) return;
    uint32_t w4[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) w4[k] = (g >= sh.groups && 4 * g + k < sh.words) ? __ldg(words + 4 * g + k) : 0u;
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
        if ((g / 32u) % 8u != r) continue;
        if (g >= sh.groups) q[r] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
        const uint32_t keep = sh.last_bits ? (1u << sh.last_bits) - 1u : 0xffffffffu;
        const uint32_t last = (sh.words - 1u) & 3u;
        if (last == 0) q[r].x &= keep;
        if (last == 1) q[r].y &= keep;
        if (last == 2) q[r].z &= keep;
        if (last == 3) q[r].w &= keep;
    }
}

// This warp's 8 rows (32 uint4 each) of block `bl` of `col`, read from global memory: bits and words
// past the column's end read 0. All loads are in flight together (at a column's end too: a branch
// per row made the last block of a column wait for its rows one after another). A mask that starts
// inside a 16-byte group (4-byte aligned) is read word by word.
template <typename Col>
__device__ __forceinline__ void popc_block_load(const Col& col, uint64_t bl, const PopcShare& sh, uint32_t warp,
                                                uint32_t lane, uint4 (&q)[8])
{
    const uint32_t* __restrict__ words = col.mask + bl * ((1u << SCAN_BLOCK_LOG2) / 32);
    if ((reinterpret_cast<uintptr_t>(col.mask) & 15u) == 0) {
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {
            const uint32_t v = (warp * 8 + r) * 32 + lane;
            q[r] = make_uint4(0u, 0u, 0u, 0u);
            if (v < sh.groups) q[r] = __ldg(reinterpret_cast<const uint4*>(words) + v);
        }
        if (4u * sh.groups != sh.words || sh.last_bits) popc_mask_end(words, sh, warp, lane, q);
        return;
    }
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
        uint32_t w4[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t w = ((warp * 8 + r) * 32 + lane) * 4 + k;
            w4[k] = w < sh.words ? __ldg(words + w) : 0u;
            if (w == sh.words - 1u && sh.last_bits) w4[k] &= (1u << sh.last_bits) - 1u;
        }
        q[r] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
    }
}

// The rest of a block once every warp holds its rows in q: chunk offsets within the block,
// the block sum, the sparse hint (sparse_seen) and, in the hybrid form, the sparse-unit
// marks. Called by all 256 threads; returns after a barrier, so s_warp may be rewritten.
// s_epoch (written by thread 0 before its first call) is read after the first barrier here.
template <int LPC, typename Col>
__device__ __forceinline__ void popc_block_finish(const BlockScanParams& p, const Col& col, uint64_t blk,
                                                  uint64_t bl, const uint4 (&q)[8], uint32_t* s_warp,
                                                  uint32_t* s_whalf, const uint32_t* s_epoch, uint32_t& sparse_seen)
{
    constexpr uint32_t CHUNK_LOG2 = LPC == 1 ? 7 : LPC == 2 ? 8 : LPC == 4 ? 9 : LPC == 8 ? 10 : LPC == 16 ? 11 : 12;
    static_assert((1u << CHUNK_LOG2) == LPC * 128u, "chunk length = 128 elements per lane");
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint64_t n = col.n;
    const uint64_t nchunks = (n + (1ull << CHUNK_LOG2) - 1) >> CHUNK_LOG2;
    const uint64_t row0 = bl * 64 + warp * 8;
    uint32_t rel[8]; // offset of this lane's chunk within the warp's 8 rows
    uint32_t run = 0, half = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint32_t c = __popc(q[r].x) + __popc(q[r].y) + __popc(q[r].z) + __popc(q[r].w);
        if constexpr (LPC == 32) {
            // a chunk is a whole row: its offset is the run before it, its count one reduction
            rel[r] = run;
            run += __reduce_add_sync(0xffffffffu, c);
            if (r == 3) half = run;
            continue;
        }
        const uint32_t incl = warp_incl_scan(c, lane);
        // the chunk's in-row offset: the exclusive scan at its first lane
        const uint32_t ex = __shfl_sync(0xffffffffu, incl - c, lane & ~static_cast<uint32_t>(LPC - 1));
        rel[r] = run + ex;
        run += __shfl_sync(0xffffffffu, incl, 31);
        if (r == 3) half = run;
    }
    // sparse hint over the warp's two aligned 16K-element groups (rows 0-3, 4-7), whole ones only: the short
    // end of a column has few selected elements at any selectivity, and the gather costs a column without
    // sparse units 5 us (1.4 x 2^22 u32, half selected, ending 631 elements into a group: 20.7 -> 15.4)
    sparse_seen += (half <= 512u) && (row0 + 4) * 4096 <= n;
    sparse_seen += (run - half <= 512u) && (row0 + 8) * 4096 <= n;
    if (lane == 0) {
        s_warp[warp] = run;
        s_whalf[warp] = half;
    }
    __syncthreads();
    if (p.item_flags) mark_sparse_units(p, col, bl, s_warp, s_whalf, *s_epoch);
    uint32_t wbase = 0, btot = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const uint32_t v = s_warp[w];
        wbase += (static_cast<uint32_t>(w) < warp) ? v : 0u;
        btot += v;
    }
    if ((lane & static_cast<uint32_t>(LPC - 1)) == 0u) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint64_t chunk = ((row0 + r) * 32 + lane) / LPC;
            if (chunk < nchunks) col.offsets[chunk] = wbase + rel[r];
        }
    }
    if (tid == 0) p.blk_sum[blk] = btot;
    __syncthreads(); // s_warp is rewritten by the next block
}

// The writeout gathers the sparse units instead of reading them whole if at least SPARSE_GROUPS_MIN of the pass's
// groups are sparse, and half of them (long columns of 4- and 8-byte elements, and large plans: one in 12). Where
// the lines lie (3-pass calls on B200, us, gathering / reading whole): all groups sparse (p = 0.01) 2^21 u32 (128
// groups) 10.0 / 8.6, 2^22 11.3 / 11.5, 2^23 12.0 / 14.2, u64 11.4 / 17.8; runs of 65536 (less than half) 2^24 u8 47 / 18,
// u32 33 / 26, 2^27 u8 110 / 61, u32 125 / 125; 2^27 u32 with its last fifth empty 170 / 181, its last tenth 183 / 188;
// plans of 40 columns and 8 MB with a few sparse ones 29.8 / 14.8, 128 columns and 470 MB 159 / 143.
constexpr uint64_t SPARSE_GROUPS_MIN = 256;
constexpr uint64_t LONG_BLOCKS = 256; // 2^26 elements

// The end of both pass-1+2 kernels (all threads): the finishing ticket carries in its upper 20 bits how many
// of the 16 groups of the CTA's average block are sparse, in sixteenths (in whole groups an evenly spread share
// loses up to half of itself), so the last CTA learns their share from its own atomic (no array to read).
// The last CTA scans the block sums and closes the epoch; the call's scan is marked clean unless a CTA
// poisoned this epoch. sparse_seen: this warp's sparse groups, of `blocks` blocks; s_warp: free.
__device__ __forceinline__ void popc_blocks_finish_grid(const BlockScanParams& p, uint32_t sparse_seen, uint32_t blocks,
                                                        uint32_t* s_warp, const uint32_t* s_epoch, uint32_t* s_flag,
                                                        uint64_t* s_scan, uint64_t* s_prefix, uint64_t prefix_room)
{
    const uint32_t tid = threadIdx.x;
    if ((tid & 31u) == 0) s_warp[tid >> 5] = sparse_seen;
    __syncthreads();
    const uint32_t epoch = *s_epoch; // written by thread 0 before the barrier above
    if (tid == 0) {
        uint32_t groups = 0;
        for (uint32_t w = 0; w < 8; ++w) groups += s_warp[w];
        // at most 256, of at most 2048 CTAs, which 12 bits count
        const uint32_t mean = static_cast<uint32_t>(__fdividef(static_cast<float>(groups) * 16.0f, static_cast<float>(blocks)) + 0.01f);
        __threadfence(); // this CTA's offsets and block sums before its ticket
        const uint32_t prev = atomicAdd(&p.hdr->scan_done_counter, 1u + (mean << 12));
        const bool last = (prev & 0xfffu) == gridDim.x - 1;
        const uint64_t sum = (prev >> 12) + mean;
        const uint32_t share = p.num_blocks > LONG_BLOCKS && (p.cols || p.col0.elem_bytes >= 4) ? 12u : 2u;
        const bool sparse = sum * share >= 256u * gridDim.x && sum * p.num_blocks >= 16u * SPARSE_GROUPS_MIN * gridDim.x;
        *s_flag = last ? (1u | (sparse ? 2u : 0u)) : 0u;
    }
    __syncthreads();
    const uint32_t fin = *s_flag;
    if (!(fin & 1u)) return;
    __threadfence(); // every other CTA's block sums (and any poison mark) are visible
    const bool clean = reinterpret_cast<volatile ws_header*>(p.hdr)->poison_epoch != epoch;
    blocks_last_cta(p, s_scan, clean, s_prefix, prefix_room);
    epilogue_last_blocks(p.hdr, epoch, (fin & 2u) != 0u, p.keep_begin, p.keep_end, clean, p.cols == nullptr);
}

template <int LPC>
__global__ void __launch_bounds__(256, 4) k_popc_blocks(const BlockScanParams p)
{
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_whalf[8];
    __shared__ uint64_t s_scan[8];
    __shared__ uint64_t s_prefix[1024];
    __shared__ uint32_t s_flag;
    __shared__ uint32_t s_epoch;
    const uint32_t tid = threadIdx.x;
    grid_dependency_wait(); // earlier calls may still be using this workspace
    if (tid == 0) s_epoch = p.hdr->epoch;
    uint32_t sparse_seen = 0;
    uint32_t blocks = 0;
    for (uint64_t blk = blockIdx.x; blk < p.num_blocks; blk += gridDim.x, ++blocks) {
        const ColumnDesc& col = column_of(p.col0, p.cols, p.blk_col, blk);
        const uint64_t bl = blk - col.tile_base; // block within its column
        uint4 q[8];
        popc_block_load(col, bl, popc_share(col, bl), tid >> 5, tid & 31u, q);
        popc_block_finish<LPC>(p, col, blk, bl, q, s_warp, s_whalf, &s_epoch, sparse_seen);
    }
    popc_blocks_finish_grid(p, sparse_seen, blocks, s_warp, &s_epoch, &s_flag, s_scan, s_prefix, 1024);
}

// ---------------------------------------------------------------------------------
// Pass 1 + 2, streaming form for long masks (more than 4 blocks per SM, where the
// register-staged k_popc_blocks needs a second round of CTAs and pays the load latency and
// the tail of a round twice). POPC_STREAM_CTAS CTAs per SM each take a contiguous range of
// blocks; thread 0 streams them through POPC_STAGES shared-memory stages of 32 KB with 1-D
// bulk copies (cp.async.bulk, no multicast), so the next block of every CTA is in flight
// while its warps count the current one. A stage is refilled once every warp has left the
// block it held (the barrier that ends popc_block_finish). Of a column's last block the whole
// 16-byte groups are copied, and the words after them (all words of a mask that starts inside such
// a group) written into the stage by the threads. The per-block work and the end are those of k_popc_blocks.
// The shape was measured on B200 at 2^28 f32 and 2^29 u8/u16 (3-pass calls, us per call):
// 3 CTAs x 2 stages beat 1 x 6 (the counting of one CTA's 8 warps is latency-bound, so one
// CTA per SM left the copies waiting on it), 2 x 3 and 4 x 1. All blocks are counted by the same
// code out of the stage: with a second source (global memory, for a column's last block) the
// registers of both met at the count, and the kernel, alone, took 39 us instead of 25 for the 1470
// blocks of 256 uneven columns.
// A stage wait that runs out records DEVERR_PIPELINE_TIMEOUT and poisons the call's scan;
// the CTA then issues no further copies and waits (bounded) for the ones in flight.
// ---------------------------------------------------------------------------------
#ifndef CS_POPC_STAGES
#define CS_POPC_STAGES 2
#endif
#ifndef CS_POPC_STREAM_CTAS
#define CS_POPC_STREAM_CTAS 3
#endif
constexpr uint32_t POPC_STAGES = CS_POPC_STAGES;
constexpr int POPC_STREAM_CTAS = CS_POPC_STREAM_CTAS; // CTAs per SM
constexpr uint32_t MASK_BLOCK_BYTES = (1u << SCAN_BLOCK_LOG2) / 8; // 32 KB of mask per block
constexpr uint64_t POPC_WAIT_NS = 2000000000ull; // bound on one stage wait (a copy lands in microseconds)
constexpr uint32_t POPC_STREAM_SMEM = POPC_STAGES * MASK_BLOCK_BYTES;

// What the copy left out of a block, into its stage: the words past the whole groups, with the bits
// past the column's end cleared, and zeros after them. All 256 threads.
__device__ __forceinline__ void popc_fill_rest(const uint32_t* words, const PopcShare& sh, uint4* stage)
{
    const uint32_t keep = sh.last_bits ? (1u << sh.last_bits) - 1u : 0xffffffffu;
    uint32_t* sw = reinterpret_cast<uint32_t*>(stage);
    constexpr uint32_t WORDS = MASK_BLOCK_BYTES / 4;
    if (4u * sh.groups == sh.words && threadIdx.x == 0) sw[sh.words - 1u] &= keep;
#pragma unroll 8
    for (uint32_t w = 4u * sh.groups + threadIdx.x; w < WORDS; w += 256) {
        uint32_t x = w < sh.words ? __ldg(words + w) : 0u;
        if (w == sh.words - 1u) x &= keep;
        sw[w] = x;
    }
}

// What k_popc_stream needs of the column that a block belongs to. In a plan a CTA keeps these of its
// next blocks in shared memory, read by all its threads at once: finding a block's column is two
// dependent loads, which thread 0 otherwise made before each copy and every warp before each block.
struct PopcBlock {
    const uint32_t* mask;
    uint64_t* offsets;
    uint64_t n;
    uint64_t bl; // block within its column
    uint64_t item_base;
    uint32_t elem_bytes;
};
constexpr uint32_t POPC_TABLE = 64; // blocks; refilled by halves

template <int LPC>
__global__ void __launch_bounds__(256, POPC_STREAM_CTAS) k_popc_stream(const BlockScanParams p)
{
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t s_full[POPC_STAGES];
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_whalf[8];
    __shared__ uint64_t s_scan[8];
    __shared__ uint32_t s_flag;
    __shared__ uint32_t s_epoch;
    __shared__ uint32_t s_fail;
    __shared__ PopcBlock s_block[POPC_TABLE];
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint64_t b0 = blockIdx.x * p.num_blocks / gridDim.x;
    const uint64_t b1 = (blockIdx.x + 1ull) * p.num_blocks / gridDim.x;
    if (tid == 0) {
        for (uint32_t s = 0; s < POPC_STAGES; ++s) mbar_init(&s_full[s], 1);
        fence_mbar_init();
        s_fail = 0u;
    }
    grid_dependency_wait(); // the mask may come from the previous kernel, the workspace too
    // blocks [from, from + count) of this CTA into the table
    auto describe = [&](uint64_t from, uint32_t count) {
        if (tid >= count || from + tid >= b1) return;
        const uint64_t blk = from + tid;
        const ColumnDesc& c = p.cols[__ldg(p.blk_col + blk)];
        s_block[(blk - b0) % POPC_TABLE] = PopcBlock{c.mask, c.offsets, c.n, blk - c.tile_base, c.item_base, c.elem_bytes};
    };
    auto block_at = [&](uint64_t blk) -> PopcBlock {
        if (p.cols) return s_block[(blk - b0) % POPC_TABLE];
        return PopcBlock{p.col0.mask, p.col0.offsets, p.col0.n, blk, 0, p.col0.elem_bytes};
    };
    // a block's whole 16-byte groups are copied in bulk, if it has any
    uint32_t pending = 0; // thread 0: stages with a copy in flight
    auto issue = [&](uint64_t blk, uint32_t s) {
        const PopcBlock c = block_at(blk);
        const uint32_t bytes = popc_share(c, c.bl).groups * 16u;
        if (bytes == 0) return;
        mbar_arrive_expect_tx(&s_full[s], bytes);
        bulk_g2s(smem + s * MASK_BLOCK_BYTES, c.mask + c.bl * (MASK_BLOCK_BYTES / 4), bytes, &s_full[s]);
        pending |= 1u << s;
    };
    if (p.cols) {
        describe(b0, POPC_TABLE);
        __syncthreads();
    }
    if (tid == 0) {
        // the first copies go out before the header read (thread 0 initialised the barriers)
        for (uint32_t k = 0; k < POPC_STAGES && b0 + k < b1; ++k) issue(b0 + k, k);
        s_epoch = p.hdr->epoch;
    }
    __syncthreads(); // barriers initialised, s_epoch and s_fail visible
    const uint32_t epoch = s_epoch;
    uint32_t sparse_seen = 0;
    uint32_t parity = 0; // bit s: parity of the phase stage s completes next
    for (uint64_t i = 0; b0 + i < b1; ++i) {
        const uint64_t blk = b0 + i;
        const uint32_t s = static_cast<uint32_t>(i % POPC_STAGES);
        const PopcBlock col = block_at(blk);
        const uint64_t bl = col.bl;
        // the half of the table whose blocks are done (the barrier ending popc_block_finish)
        if (p.cols && i != 0 && i % (POPC_TABLE / 2) == 0) describe(blk + POPC_TABLE / 2, POPC_TABLE / 2);
        const PopcShare sh = popc_share(col, bl);
        uint4* sv = reinterpret_cast<uint4*>(smem + s * MASK_BLOCK_BYTES);
        // after a failure no stage is refilled, so nothing more is waited for
        if (sh.groups != 0u && *reinterpret_cast<volatile uint32_t*>(&s_fail) == 0u) {
            if (mbar_wait_bounded(&s_full[s], (parity >> s) & 1u, POPC_WAIT_NS)) {
                parity ^= 1u << s;
                if (tid == 0) pending &= ~(1u << s);
            } else {
                atomicOr(&s_fail, 1u);
                if (lane == 0) {
                    record_error(p.hdr, DEVERR_PIPELINE_TIMEOUT);
                    reinterpret_cast<volatile ws_header*>(p.hdr)->poison_epoch = epoch;
                }
            }
        }
        // the rest of the block into the stage, so that all blocks are counted by the same code
        if (sh.groups != MASK_BLOCK_BYTES / 16 || sh.last_bits != 0u) {
            popc_fill_rest(col.mask + bl * (MASK_BLOCK_BYTES / 4), sh, sv);
            fence_proxy_async(); // before the next copy into this stage
            __syncthreads();
        }
        uint4 q[8];
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) q[r] = sv[(warp * 8 + r) * 32 + lane];
        popc_block_finish<LPC>(p, col, blk, bl, q, s_warp, s_whalf, &s_epoch, sparse_seen);
        // every warp has left stage s (the barrier ending popc_block_finish): refill it
        if (tid == 0 && b0 + i + POPC_STAGES < b1 && s_fail == 0u) issue(b0 + i + POPC_STAGES, s);
    }
    // after a failed wait: the copies still in flight (each stage's pending phase is the one
    // `parity` names) must land before the CTA exits
    if (tid == 0 && pending != 0u) {
        for (uint32_t s = 0; s < POPC_STAGES; ++s)
            if ((pending >> s) & 1u) mbar_wait_bounded(&s_full[s], (parity >> s) & 1u, POPC_WAIT_NS);
    }
    // (no copy is in flight any more: the stages hold the block prefixes)
    popc_blocks_finish_grid(p, sparse_seen, static_cast<uint32_t>(b1 - b0), s_warp, &s_epoch, &s_flag, s_scan, reinterpret_cast<uint64_t*>(smem),
                            POPC_STREAM_SMEM / 8);
}

// Masks of more than this many blocks per SM take the streaming form.
#ifndef CS_POPC_STREAM_BLOCKS_PER_SM
#define CS_POPC_STREAM_BLOCKS_PER_SM 4
#endif

namespace {
constexpr int POPC_MAX_DEVICES = 64;
unsigned g_popc_stream_attr[POPC_MAX_DEVICES]; // bit k: smem attribute of variant k applied

template <int LPC>
cudaError_t launch_popc_stream(const BlockScanParams& p, uint32_t grid, cudaStream_t stream, int variant)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned bit = 1u << variant;
    const bool known = dev >= 0 && dev < POPC_MAX_DEVICES;
    if (!known || !(__atomic_load_n(&g_popc_stream_attr[dev], __ATOMIC_ACQUIRE) & bit)) {
        e = cudaFuncSetAttribute(k_popc_stream<LPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(POPC_STREAM_SMEM));
        if (e != cudaSuccess) return e;
        if (known) __atomic_fetch_or(&g_popc_stream_attr[dev], bit, __ATOMIC_RELEASE);
    }
    return launch_pdl(k_popc_stream<LPC>, dim3(grid), dim3(256), POPC_STREAM_SMEM, stream, p);
}
} // namespace

cudaError_t launch_popc_blocks(const BlockScanParams& p, int num_sms, cudaStream_t stream)
{
    cudaError_t e;
    if (num_sms > 0 && p.num_blocks > static_cast<uint64_t>(num_sms) * CS_POPC_STREAM_BLOCKS_PER_SM) {
        const uint32_t grid = static_cast<uint32_t>(num_sms) * POPC_STREAM_CTAS; // fewer CTAs than blocks
        switch (p.chunk_log2) {
            case 7: e = launch_popc_stream<1>(p, grid, stream, 0); break;
            case 8: e = launch_popc_stream<2>(p, grid, stream, 1); break;
            case 9: e = launch_popc_stream<4>(p, grid, stream, 2); break;
            case 10: e = launch_popc_stream<8>(p, grid, stream, 3); break;
            case 11: e = launch_popc_stream<16>(p, grid, stream, 4); break;
            case 12: e = launch_popc_stream<32>(p, grid, stream, 5); break;
            default: return cudaErrorInvalidValue;
        }
        note_launch();
        return e;
    }
    uint64_t blocks = p.num_blocks;
    uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
    if (cap > POPC_FLAG_SLOTS) cap = POPC_FLAG_SLOTS;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    const dim3 g(static_cast<unsigned>(blocks)), b(256);
    switch (p.chunk_log2) {
        case 7: e = launch_pdl(k_popc_blocks<1>, g, b, 0, stream, p); break;
        case 8: e = launch_pdl(k_popc_blocks<2>, g, b, 0, stream, p); break;
        case 9: e = launch_pdl(k_popc_blocks<4>, g, b, 0, stream, p); break;
        case 10: e = launch_pdl(k_popc_blocks<8>, g, b, 0, stream, p); break;
        case 11: e = launch_pdl(k_popc_blocks<16>, g, b, 0, stream, p); break;
        case 12: e = launch_pdl(k_popc_blocks<32>, g, b, 0, stream, p); break;
        default: return cudaErrorInvalidValue;
    }
    note_launch();
    return e;
}

// ---------------------------------------------------------------------------------
// Pass 3, alignment-agnostic form: one warp per chunk walks the chunk's mask words; lane
// l owns element 32*w + l, its output slot is popc(word & lanemask_lt) past the running
// offset. Empty chunks are skipped using the pass-1 counts. Mirrors the reference's
// warp-cooperative writeout (kernel_3pass_proc_true_striding_naive_writeout,
// src/kernels/kernel_3pass.cuh:216-327) with LSB-first bits and 64-bit indexing.
// ---------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_writeout_naive(const T* __restrict__ in, const uint32_t* __restrict__ mask,
                                                        T* __restrict__ out, uint64_t n,
                                                        const uint64_t* __restrict__ chunk_offsets,
                                                        const uint32_t* __restrict__ chunk_counts, uint32_t chunk_log2,
                                                        const ws_header* hdr)
{
    __shared__ uint32_t s_hflags;
    if (!(cta_header_flags(hdr, &s_hflags) & 1u)) return; // pass 2 offsets not trustworthy: write nothing
    const uint64_t nw = (n + 31) / 32;
    const uint64_t num_chunks = (n + (1ull << chunk_log2) - 1) >> chunk_log2;
    const uint64_t wpc = 1ull << (chunk_log2 - 5);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t warp_global = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t total_warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t chunk = warp_global; chunk < num_chunks; chunk += total_warps) {
        if (chunk_counts && chunk_counts[chunk] == 0u) continue;
        uint64_t pos = chunk_offsets[chunk];
        if (pos == POISON) continue;
        const uint64_t w_end = (chunk + 1) * wpc < nw ? (chunk + 1) * wpc : nw;
        for (uint64_t wi = chunk * wpc; wi < w_end; ++wi) {
            const uint32_t m = load_mask_word(mask, wi, nw, n);
            if (m == 0u) continue;
            if ((m >> lane) & 1u) out[pos + __popc(m & lt)] = in[wi * 32 + lane];
            pos += __popc(m);
        }
    }
}

cudaError_t launch_writeout_naive(const void* in, const uint32_t* mask, void* out, uint64_t n, uint32_t elem_bytes,
                                  const uint64_t* chunk_offsets, const uint32_t* chunk_counts, uint32_t chunk_log2,
                                  const ws_header* hdr, int num_sms, cudaStream_t stream)
{
    const uint64_t num_chunks = (n + (1ull << chunk_log2) - 1) >> chunk_log2;
    uint64_t blocks = (num_chunks + 7) / 8;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 8;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    const unsigned g = static_cast<unsigned>(blocks);
    switch (elem_bytes) {
        case 1:
            k_writeout_naive<uint8_t><<<g, 256, 0, stream>>>(static_cast<const uint8_t*>(in), mask,
                                                             static_cast<uint8_t*>(out), n, chunk_offsets,
                                                             chunk_counts, chunk_log2, hdr);
            break;
        case 2:
            k_writeout_naive<uint16_t><<<g, 256, 0, stream>>>(static_cast<const uint16_t*>(in), mask,
                                                              static_cast<uint16_t*>(out), n, chunk_offsets,
                                                              chunk_counts, chunk_log2, hdr);
            break;
        case 4:
            k_writeout_naive<uint32_t><<<g, 256, 0, stream>>>(static_cast<const uint32_t*>(in), mask,
                                                              static_cast<uint32_t*>(out), n, chunk_offsets,
                                                              chunk_counts, chunk_log2, hdr);
            break;
        case 8:
            k_writeout_naive<uint64_t><<<g, 256, 0, stream>>>(static_cast<const uint64_t*>(in), mask,
                                                              static_cast<uint64_t*>(out), n, chunk_offsets,
                                                              chunk_counts, chunk_log2, hdr);
            break;
        default: return cudaErrorInvalidValue;
    }
    note_launch();
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Workspace init: zero everything, then write the header.
// ---------------------------------------------------------------------------------
__global__ void k_ws_init(ws_header* hdr, uint64_t ws_bytes)
{
    uint4* p = reinterpret_cast<uint4*>(hdr);
    const uint64_t n16 = ws_bytes / 16u;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n16; i += stride)
        p[i] = make_uint4(0, 0, 0, 0);
}

__global__ void k_ws_header(ws_header* hdr, uint64_t ws_bytes)
{
    hdr->magic = WS_MAGIC;
    hdr->epoch = EPOCH_MIN;
    hdr->err = 0;
    hdr->tile_counter = 0;
    hdr->done_counter = 0;
    hdr->scan_tile_counter = 0;
    hdr->scan_done_counter = 0;
    hdr->ws_bytes = ws_bytes;
}

cudaError_t launch_ws_init(ws_header* hdr, size_t ws_bytes, cudaStream_t stream)
{
    uint64_t blocks = (ws_bytes / 16 + 255) / 256;
    if (blocks > 1024) blocks = 1024;
    if (blocks == 0) blocks = 1;
    k_ws_init<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(hdr, ws_bytes);
    k_ws_header<<<1, 1, 0, stream>>>(hdr, ws_bytes);
    note_launch(2);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Seeded generators. mix64 is the SplitMix64 output function (Steele, Lea, Flood 2014)
// applied to seed + (i+1)*golden-gamma, so element i depends only on (seed, i).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t seed, uint64_t i)
{
    uint64_t z = seed + (i + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

template <typename T>
__global__ void k_gen_payload(T* out, uint64_t n, uint64_t seed, int float_unit)
{
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t h = mix64(seed, i);
        if (sizeof(T) == 4 && float_unit) {
            const float f = static_cast<float>(static_cast<uint32_t>(h >> 40)) * (1.0f / 16777216.0f);
            out[i] = static_cast<T>(__float_as_uint(f));
        } else {
            out[i] = static_cast<T>(h);
        }
    }
}

cudaError_t launch_gen_payload(void* out, uint64_t n, uint32_t elem_bytes, uint64_t seed, int float_unit, int num_sms,
                               cudaStream_t stream)
{
    uint64_t blocks = (n + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    const unsigned g = static_cast<unsigned>(blocks);
    switch (elem_bytes) {
        case 1: k_gen_payload<uint8_t><<<g, 256, 0, stream>>>(static_cast<uint8_t*>(out), n, seed, 0); break;
        case 2: k_gen_payload<uint16_t><<<g, 256, 0, stream>>>(static_cast<uint16_t*>(out), n, seed, 0); break;
        case 4: k_gen_payload<uint32_t><<<g, 256, 0, stream>>>(static_cast<uint32_t*>(out), n, seed, float_unit); break;
        case 8: k_gen_payload<uint64_t><<<g, 256, 0, stream>>>(static_cast<uint64_t*>(out), n, seed, 0); break;
        default: return cudaErrorInvalidValue;
    }
    note_launch();
    return cudaGetLastError();
}

// word w packs elements 32w..32w+31, LSB-first; bit set iff (mix64(seed, i) >> 32) < threshold
__global__ void k_gen_mask_bernoulli(uint32_t* mask, uint64_t n, uint64_t threshold, uint64_t seed)
{
    const uint64_t nw = (n + 31) / 32;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < nw; w += stride) {
        uint32_t m = 0;
        for (uint32_t b = 0; b < 32; ++b) {
            const uint64_t i = w * 32 + b;
            if (i < n && (mix64(seed, i) >> 32) < threshold) m |= 1u << b;
        }
        mask[w] = m;
    }
}

cudaError_t launch_gen_mask_bernoulli(uint32_t* mask, uint64_t n, uint64_t threshold, uint64_t seed, int num_sms,
                                      cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    uint64_t blocks = (nw + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_gen_mask_bernoulli<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, n, threshold, seed);
    note_launch();
    return cudaGetLastError();
}

// Alternating runs, step 1: toggle words (bit i set iff position i starts a new run),
// stored as their in-word prefix parity, plus per-word toggle popcounts for the scan.
__global__ void k_gen_runs_toggle(uint32_t* mask, uint32_t* parity_counts, uint64_t n, uint64_t threshold, uint64_t seed)
{
    const uint64_t nw = (n + 31) / 32;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < nw; w += stride) {
        uint32_t t = 0;
        for (uint32_t b = 0; b < 32; ++b) {
            const uint64_t i = w * 32 + b;
            if (i < n && (mix64(seed, i) >> 32) < threshold) t |= 1u << b;
        }
        parity_counts[w] = static_cast<uint32_t>(__popc(t));
        uint32_t x = t; // bit j <- xor of bits 0..j
        x ^= x << 1;
        x ^= x << 2;
        x ^= x << 4;
        x ^= x << 8;
        x ^= x << 16;
        mask[w] = x;
    }
}

cudaError_t launch_gen_runs_toggle(uint32_t* mask, uint32_t* parity_counts, uint64_t n, uint64_t threshold,
                                   uint64_t seed, int num_sms, cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    uint64_t blocks = (nw + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_gen_runs_toggle<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, parity_counts, n, threshold, seed);
    note_launch();
    return cudaGetLastError();
}

// Alternating runs, step 2: flip a word when an odd number of toggles precede it.
__global__ void k_gen_runs_apply(uint32_t* mask, const uint64_t* parity_offsets, uint64_t n)
{
    const uint64_t nw = (n + 31) / 32;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < nw; w += stride) {
        uint32_t m = mask[w];
        if (parity_offsets[w] & 1ull) m = ~m;
        if (w == nw - 1 && (n & 31u)) m &= (1u << (n & 31u)) - 1u;
        mask[w] = m;
    }
}

cudaError_t launch_gen_runs_apply(uint32_t* mask, const uint64_t* parity_offsets, uint64_t n, int num_sms,
                                  cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    uint64_t blocks = (nw + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_gen_runs_apply<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, parity_offsets, n);
    note_launch();
    return cudaGetLastError();
}

__global__ void k_gen_mask_dense_prefix(uint32_t* mask, uint64_t n, uint64_t k)
{
    const uint64_t nw = (n + 31) / 32;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < nw; w += stride) {
        const uint64_t lo = w * 32;
        uint32_t m;
        if (lo + 32 <= k) m = 0xffffffffu;
        else if (lo >= k) m = 0u;
        else m = (1u << (k - lo)) - 1u;
        mask[w] = m;
    }
}

cudaError_t launch_gen_mask_dense_prefix(uint32_t* mask, uint64_t n, uint64_t k, int num_sms, cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    uint64_t blocks = (nw + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_gen_mask_dense_prefix<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, n, k);
    note_launch();
    return cudaGetLastError();
}

// Periodic mask: bit i = bit (i % L) of pattern (the selection of compressstore_pattern as
// a mask in memory; the reference builds it MSB-first on the host, generate_mask_pattern,
// src/data_generator.cuh:113-128).
__global__ void k_gen_mask_pattern(uint32_t* mask, uint64_t n, uint32_t pattern, uint32_t L)
{
    const uint64_t nw = (n + 31) / 32;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < nw; w += stride) {
        uint32_t m = 0;
        uint32_t ph = static_cast<uint32_t>((w * 32) % L);
#pragma unroll 4
        for (uint32_t b = 0; b < 32; ++b) {
            m |= ((pattern >> ph) & 1u) << b;
            if (++ph == L) ph = 0;
        }
        const uint64_t lo = w * 32;
        if (lo + 32 > n) m &= (1u << (n - lo)) - 1u;
        mask[w] = m;
    }
}

cudaError_t launch_gen_mask_pattern(uint32_t* mask, uint64_t n, uint32_t pattern, uint32_t L, int num_sms,
                                    cudaStream_t stream)
{
    const uint64_t nw = (n + 31) / 32;
    uint64_t blocks = (nw + 255) / 256;
    const uint64_t cap = static_cast<uint64_t>(num_sms) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    k_gen_mask_pattern<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(mask, n, pattern, L);
    note_launch();
    return cudaGetLastError();
}

} // namespace cs
