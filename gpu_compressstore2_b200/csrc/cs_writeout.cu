// cs_writeout.cu — pass 3 of the 3-pass form (chunk length at most 4096): every warp compacts
// items of its own, without barriers, rings or other warps.
//
// DENSE ITEMS. An item is 4 KB of payload: 4 rows of 32 bytes per lane, each one 256-bit load, so
// that a lane holds consecutive elements and its mask bits are one byte, half word or word. A
// warp loads the next item's mask while it works on the present one, so the payload loads of an
// item are issued at once and lanes without a selected element issue none. Positions come
// from a packed warp scan of the lanes' counts (two rows per scan) behind the item's offset from
// pass 2; selected elements go to a stage of the warp in shared memory, and the stage leaves as
// 16-byte streaming stores.
//   * 2-, 4- and 8-byte elements: one predicated store per element, the address advancing
//     with it.
//   * 1-byte elements: four at a time are packed in registers by a byte permute whose selectors
//     come from a 16-entry table (one copy per lane, so its reads do not conflict), appended to
//     the lane's current word with funnel shifts, and stored when a word is full. The bytes of
//     a lane's last, partial word follow after a warp barrier: the next lane's first word
//     carries zeros in their place. One store per 4 selected bytes instead of one per byte:
//     the shared-memory pipe was what bound the per-byte form (75% busy).
//
// SPARSE UNITS. Units (128 KB of payload) with at most 1/32 selected are gathered instead: DRAM
// traffic is then the mask plus the sectors holding selected elements. What bounds this is
// latency (a flag, then the mask, then the payload) and, at 1% and above, DRAM sectors. Pass 1
// marks the 16K-element items of such units; a warp loads the masks of a whole item at once (128
// consecutive elements per lane and 4096-element group), writes the indices of its selected
// elements to a list in its stage at their ranks, and gathers from the list with
// SPARSE_INFLIGHT loads per lane in flight before the first store; a load fetches 64 bytes
// instead of a line (ldg_gather). When there are fewer items than warps a warp takes
// one group, so that a column with few sparse units still spreads over many warps. The dense
// part skips exactly these units (same count test); it looks at 32 of its items at a time.
//
// What bounds the dense part is HBM at half the rows and above for 4 and 8 bytes (2^26 u32
// p = 0.5: 63.4 us, 410 MB: 6470 GB/s) and, for 1 byte, the packing (61 % of the issue slots used). Per 3-pass call
// on B200 against the TMA-staged writeout it replaces (persistent CTAs, payload tiles and masks
// through shared-memory rings, 16 compute warps in step): 2^29 u8 p = 0.5 268 -> 195 us, p = 0.9
// 332 -> 213, 2^28 u16 p = 0.5 179 -> 158, 2^28 f32 p = 0.1 247 -> 212, p = 0.5 304 -> 268, p = 0.9
// 367 -> 345, 2^27 u64 p = 0.5 269 -> 255, p = 0.9 373 -> 359, 2^24 u32 p = 0.5 30.5 -> 23. Long runs
// of calls are held back by the power limit, which is where the fewer instructions per
// element count at 4 and 8 bytes. The gather against a lane walking its mask word's bits, whose
// every load waited for the store before it: 2^28 f32 p = 0.01 95.6 -> 64, p = 0.001 49 -> 31,
// 2^29 u8 p = 0.001 93 -> 53, 2^27 u64 p = 0.01 74.5 -> 45. 8 loads in flight instead of 4 change
// little (61.5, 31.5).
//
// Reference: kernel_3pass_proc_true_striding_optimized_writeout
// (src/kernels/kernel_3pass.cuh:329-467) stages 32 source indices per warp and gathers from
// global memory; its empty-chunk skipping is :268-288.
#include <cstdint>
#include <cuda_runtime.h>

#include "cs_internal.cuh"
#include "cs_place.cuh"

namespace cs {

namespace {

constexpr uint32_t SPARSE_LIST = 1024;                    // indices of one gather round (in the stage)
constexpr uint32_t SPARSE_INFLIGHT = 4;                   // payload loads per lane in flight
static_assert(SPARSE_LIST * 2 <= STAGE_BYTES, "the list lies in the stage");

// 8 warps per CTA and 3 CTAs per SM: 80 registers hold an item's 4 loads per lane without spills.
// More resident warps with fewer registers were slower (64 registers x 4 CTAs spill; 2 rows per
// item x 5 CTAs: 2^28 f32 p = 0.5 291 against 281 us, 2^29 u8 210 against 194), and so were fewer
// (2 CTAs: 300 and 209) and items of 8 rows (2 x 8 KB per SM-warp: 269, 194). Shifted loads of narrower
// elements than 8 bytes hold three vectors per row.
constexpr uint32_t WARPS = 8;
template <typename T, bool SHIFT>
constexpr uint32_t CTAS = SHIFT && sizeof(T) < 8 ? 2 : 3;

// Warps of a CTA that stay idle for a long column of which most is selected (by thousandths): there the
// loads in flight of 24 warps per SM hold up the writes. 3-pass call on B200, us, 24 / 21 / 18 warps: 2^27 u64
// p = 0.7 298 / 295 / 309, 0.8 348 / 333 / 314, 0.9 360 / 345 / 335, 0.99 377 / - / 347, all 371 / - / 345; 2^28 u32
// p = 0.7 303 / 310 / 331, 0.8 339 / 326 / 334, 0.9 357 / 340 / 355, 2^27 0.996 189 / 193 / 198, 0.9995 190 / 195 /
// 201, all 204 / 198 / 184, 2^26 all 106 / 104 / 97, 2^28 all 370 / 360 / 368, 2^26 u32 p = 0.9 102 / 94 / 94, but
// 2^24 29.6 / 30.6 / 31.7 (few items per warp). Narrower elements are held back by their instructions: 2^28 u16
// p = 0.9 185 / 198 / 200.
template <typename T>
__device__ __forceinline__ uint32_t idle_warps(uint64_t thousandths)
{
    if constexpr (sizeof(T) == 8) return thousandths >= 750u ? 2u : 0u;
    if constexpr (sizeof(T) == 4) return thousandths >= 1000u ? 2u : thousandths >= 850u && thousandths < 970u ? 1u : 0u;
    return 0u;
}

// 32 bytes from an address `d` bytes (1 .. 15, the same for the whole column) past a 16-byte boundary: out of
// the three 16-byte vectors that hold them, or, for 8-byte elements (d = 8), as the halves of two and the one
// between them, which need no selection (2^26 u64 p = 0.1 225 -> 97 us, 0.5 251 -> 133, 0.9 338 -> 170; and 80 registers, three CTAs per SM).
template <typename T>
__device__ __forceinline__ void ldg_shifted(const uint8_t* p, uint32_t d, uint32_t (&x)[8])
{
    if constexpr (sizeof(T) == 8) {
        const uint2 a = __ldg(reinterpret_cast<const uint2*>(p));
        const uint4 b = __ldg(reinterpret_cast<const uint4*>(p + 8));
        const uint2 c = __ldg(reinterpret_cast<const uint2*>(p + 24));
        x[0] = a.x, x[1] = a.y, x[2] = b.x, x[3] = b.y, x[4] = b.z, x[5] = b.w, x[6] = c.x, x[7] = c.y;
    } else {
        const uint4* q = reinterpret_cast<const uint4*>(p - d);
        const uint4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
        const uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
        const uint32_t s = (d & 3u) * 8u;
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            uint32_t lo = w[i], hi = w[i + 1];
            if (d >= 12u) lo = w[i + 3], hi = w[i + 4 < 12 ? i + 4 : 11];
            else if (d >= 8u) lo = w[i + 2], hi = w[i + 3];
            else if (d >= 4u) lo = w[i + 1], hi = w[i + 2];
            x[i] = sizeof(T) == 4 ? lo : __funnelshift_r(lo, hi, s); // (whole words: s = 0)
        }
    }
}

// GROUPS 4096-element groups of a sparse unit of column c, from element e0.
template <typename T, int GROUPS>
__device__ __forceinline__ void sparse_groups(const ColumnDesc& c, uint64_t e0, uint32_t chunk_log2, uint32_t lane,
                                              uint16_t* list)
{
    const uint64_t n = c.n;
    if (e0 >= n) return;
    const uint64_t nw = (n + 31) / 32;
    const uint32_t* __restrict__ mask = c.mask;
    const bool vec = (reinterpret_cast<uintptr_t>(mask) & 15u) == 0;
    uint32_t m[GROUPS][4];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
        const uint64_t w0 = e0 / 32 + g * 128ull + lane * 4u; // a multiple of 4
        if (vec && w0 + 4 <= nw) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(mask + w0));
            m[g][0] = q.x, m[g][1] = q.y, m[g][2] = q.z, m[g][3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) m[g][k] = w0 + k < nw ? __ldg(mask + w0 + k) : 0u;
        }
        if (w0 + 4 >= nw && (n & 31u)) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (w0 + k == nw - 1) m[g][k] &= (1u << (n & 31u)) - 1u;
        }
    }
    constexpr uint64_t UE = unit_elems_for(sizeof(T));
    const uint64_t pos0 = chunk_offset(c, e0 >> chunk_log2, chunk_log2); // groups start on chunk boundaries
    const uint64_t u0 = e0 & ~(UE - 1);                                  // an item never straddles units
    const uint64_t off_b = chunk_offset(c, u0 >> chunk_log2, chunk_log2);
    const uint64_t off_e = u0 + UE >= n ? *c.d_count : chunk_offset(c, (u0 + UE) >> chunk_log2, chunk_log2);
    if (off_e - off_b > UE / 32) return; // an earlier call's mark: the dense part owns the unit

    uint32_t rank[GROUPS], cnt[GROUPS]; // rank of the lane's first selected element of each group
    uint32_t total = 0;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g)
        cnt[g] = __popc(m[g][0]) + __popc(m[g][1]) + __popc(m[g][2]) + __popc(m[g][3]);
#pragma unroll
    for (int g = 0; g < GROUPS; g += 2) { // two groups (at most 4096 each) per scan
        const uint32_t second = g + 1 < GROUPS ? cnt[(g + 1) % GROUPS] : 0u;
        const uint32_t own = cnt[g] | (second << 16);
        const uint32_t incl = warp_incl_scan(own, lane);
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        rank[g] = total + ((incl - own) & 0xffffu);
        total += all & 0xffffu;
        if (g + 1 < GROUPS) {
            rank[(g + 1) % GROUPS] = total + ((incl - own) >> 16);
            total += all >> 16;
        }
    }
    const T* __restrict__ in = reinterpret_cast<const T*>(c.in) + e0;
    T* __restrict__ out = reinterpret_cast<T*>(c.out) + pos0 + lane;
    const uint16_t* const mine = list + lane;
    for (uint32_t r0 = 0; r0 < total; r0 += SPARSE_LIST) {
        // indices of ranks [r0, r0 + SPARSE_LIST)
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            uint32_t at = rank[g] - r0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t mm = m[g][k];
                while (mm) {
                    if (at < SPARSE_LIST) list[at] = static_cast<uint16_t>(g * 4096 + lane * 128 + k * 32 + __ffs(mm) - 1);
                    mm &= mm - 1;
                    ++at;
                }
            }
        }
        __syncwarp();
        const uint32_t len = total - r0 < SPARSE_LIST ? total - r0 : SPARSE_LIST;
        for (uint32_t j0 = 0; j0 < len; j0 += 32 * SPARSE_INFLIGHT) {
            T x[SPARSE_INFLIGHT];
            const uint32_t left = len - j0;
#pragma unroll
            for (uint32_t i = 0; i < SPARSE_INFLIGHT; ++i)
                if (lane + 32 * i < left) x[i] = ldg_gather(in + mine[j0 + 32 * i]);
#pragma unroll
            for (uint32_t i = 0; i < SPARSE_INFLIGHT; ++i)
                if (lane + 32 * i < left) out[r0 + j0 + 32 * i] = x[i];
        }
        __syncwarp(); // the list is rewritten by the next round or work item
    }
}

// LONG: chunks longer than an item, which may then start inside one: the selected elements of the chunk before
// it come from its mask, one vector per lane, asked for with the item's own mask. (Word by word behind the
// payload's loads: 3-pass calls at chunk 4096, us, 2^27 u64 p = 0.5 286 -> 256, 0.9 382 -> 328, 2^28 u32 0.5 297
// -> 267, 0.9 396 -> 343, 2^28 u16 0.5 168 -> 155; 2^22 u64 17.6 -> 18.2.) A kernel of its own: in the other one
// its registers cost 2^28 u32 at chunk 1024 265 -> 296.
template <typename T, bool MULTI, bool SHIFT, bool LONG>
__global__ void __launch_bounds__(WARPS * 32, CTAS<T, SHIFT>) k_writeout_warp(const WriteoutParams p)
{
    constexpr uint32_t EPL = LANE_BYTES / sizeof(T); // elements per lane and row
    constexpr uint32_t ROW = 32 * EPL;
    constexpr uint32_t ITEM = ROWS * ROW;
    constexpr uint32_t ITEM_LOG2 = sizeof(T) == 1 ? 12 : sizeof(T) == 2 ? 11 : sizeof(T) == 4 ? 10 : 9;
    static_assert(ITEM == 1u << ITEM_LOG2, "elements per item");
    constexpr uint64_t UE = unit_elems_for(sizeof(T));
    constexpr uint32_t IPU = UE / ITEM; // items per unit
    constexpr uint32_t VEC = 16 / sizeof(T);
    constexpr uint32_t NONE = 0xffffffffu;
    __shared__ __align__(128) uint8_t s_stage[WARPS][STAGE_BYTES];
    __shared__ uint32_t s_lut[sizeof(T) == 1 ? PACK_TABLE_WORDS : 1];
    __shared__ uint32_t s_hflags;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    if constexpr (sizeof(T) == 1) fill_pack_table(s_lut, WARPS * 32);
    grid_dependency_wait(); // offsets and counts of pass 2
    const uint32_t hflags = cta_header_flags(p.hdr, &s_hflags); // a barrier: the table is filled
    if (!(hflags & 1u)) return; // pass 2 offsets not trustworthy: write nothing
    const bool hybrid = p.sparse_max != 0 && (hflags & 2u) != 0u;
    uint8_t* const stage = s_stage[warp];
    const uint32_t stage_a = smem_u32(stage);
    const uint32_t lut = sizeof(T) == 1 ? smem_u32(s_lut) + lane * 4 : 0u;
    const uint32_t num_items = static_cast<uint32_t>(p.num_units) * IPU; // below 2^32 for every column the library takes
    // a long column of mostly selected elements runs better with fewer warps
    uint32_t active = MULTI ? WARPS - p.throttle : WARPS;
    if constexpr (!MULTI && sizeof(T) >= 4) {
        if (p.throttle != 0u) active -= idle_warps<T>(*p.col0.d_count * 1000 / p.col0.n);
    }
    if (sizeof(T) >= 4 && warp >= active) return;
    const uint32_t warp_global = blockIdx.x * active + warp;
    const uint32_t total_warps = gridDim.x * active;

    auto column = [&](uint32_t it) -> const ColumnDesc& {
        return MULTI ? p.cols[__ldg(p.unit_col + it / IPU)] : p.col0;
    };
    auto first_elem = [&](const ColumnDesc& C, uint32_t it) -> uint64_t {
        return static_cast<uint64_t>(MULTI ? it - static_cast<uint32_t>(C.unit_base) * IPU : it) * ITEM;
    };
    // This warp's items in turn: warp_global, warp_global + total_warps, ... In the hybrid form
    // it looks at 32 of them at a time (one per lane) and keeps those of dense units.
    uint32_t base = warp_global; // first item of the window, or the next item
    uint32_t window = 0;         // hybrid: items of the window still to be taken
    bool opened = false;
    auto next_item = [&]() -> uint32_t {
        if (!hybrid) {
            const uint32_t it = base;
            if (it >= num_items) return NONE;
            base += total_warps;
            return it;
        }
        while (window == 0u) {
            if (opened) {
                if (num_items - base <= 32u * total_warps) return NONE; // base < num_items while open
                base += 32u * total_warps;
            }
            if (base >= num_items) return NONE;
            opened = true;
            const uint64_t mine = static_cast<uint64_t>(base) + static_cast<uint64_t>(lane) * total_warps;
            bool take = mine < num_items;
            if (take) {
                const ColumnDesc& C = column(static_cast<uint32_t>(mine));
                const uint64_t u0 = first_elem(C, static_cast<uint32_t>(mine)) & ~(UE - 1);
                const uint64_t off_b = chunk_offset(C, u0 >> p.chunk_log2, p.chunk_log2);
                const uint64_t off_e =
                    u0 + UE >= C.n ? *C.d_count : chunk_offset(C, (u0 + UE) >> p.chunk_log2, p.chunk_log2);
                take = off_e - off_b > p.sparse_max;
            }
            window = __ballot_sync(0xffffffffu, take);
        }
        const uint32_t k = __ffs(window) - 1;
        window &= window - 1;
        return base + k * total_warps;
    };

    uint32_t m[ROWS]; // the present item's mask bits, loaded one item ahead
    uint4 head = make_uint4(0u, 0u, 0u, 0u); // LONG: and a lane's share of its chunk's mask before it
    auto load_mask = [&](uint32_t it) {
        const ColumnDesc& C = column(it);
        const uint64_t e0 = first_elem(C, it);
        const uint8_t* mb = reinterpret_cast<const uint8_t*>(C.mask);
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) {
            const uint64_t e = e0 + r * ROW + lane * EPL;
            uint32_t v = 0;
            if (e < C.n) {
                if constexpr (EPL == 32) v = __ldg(reinterpret_cast<const uint32_t*>(mb + (e >> 3)));
                else if constexpr (EPL == 16) v = __ldg(reinterpret_cast<const uint16_t*>(mb + (e >> 3)));
                else v = __ldg(mb + (e >> 3));
            }
            m[r] = v;
        }
        if constexpr (LONG) {
            // less than a chunk of 4096 elements: 128 words, four to a lane
            const uint64_t w0 = ((e0 >> p.chunk_log2) << p.chunk_log2) >> 5;
            head = make_uint4(0u, 0u, 0u, 0u);
            if (e0 < C.n && lane * 4u < static_cast<uint32_t>((e0 >> 5) - w0)) {
                const uint32_t* hw = C.mask + w0 + lane * 4u;
                if ((reinterpret_cast<uintptr_t>(C.mask) & 15u) == 0) head = __ldg(reinterpret_cast<const uint4*>(hw));
                else head = make_uint4(__ldg(hw), __ldg(hw + 1), __ldg(hw + 2), __ldg(hw + 3));
            }
        }
    };
    uint32_t it = next_item();
    if (it != NONE) load_mask(it);
    while (it != NONE) {
        const ColumnDesc& C = column(it);
        const uint64_t n = C.n;
        const uint64_t e0 = first_elem(C, it);
        if (e0 >= n) { // past the end of a column's last unit
            it = next_item();
            if (it != NONE) load_mask(it);
            continue;
        }
        uint32_t before = 0; // selected elements of the chunk before the item
        if constexpr (LONG) before = __reduce_add_sync(0xffffffffu, __popc(head.x) + __popc(head.y) + __popc(head.z) + __popc(head.w));
        uint32_t bits[ROWS];
        uint32_t x[ROWS][8];
        const uint8_t* src = C.in + e0 * sizeof(T) + lane * LANE_BYTES;
        const uint32_t phase = SHIFT ? static_cast<uint32_t>(reinterpret_cast<uintptr_t>(C.in) & 15u) : 0u;
        const bool in32 = (reinterpret_cast<uintptr_t>(C.in) & 31u) == 0;
        const bool whole = e0 + ITEM <= n;
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) {
            uint32_t b = m[r];
            if constexpr (EPL == 4) b = (b >> ((lane & 1u) * 4)) & 0xfu;
            const uint64_t e = e0 + r * ROW + lane * EPL;
            if (!whole && e + EPL > n) b &= e < n ? (1u << (n - e)) - 1u : 0u; // n - e < EPL <= 32
            bits[r] = b;
            if (b) {
                // a shifted load of narrower elements takes whole 16-byte vectors, which must lie inside the column
                const bool inside = SHIFT && sizeof(T) < 8 ? e > 0 && e * sizeof(T) + 48 - phase <= n * sizeof(T) : whole || e + EPL <= n;
                if (inside) {
                    if constexpr (SHIFT) ldg_shifted<T>(src + r * ROW_BYTES, phase, x[r]);
                    else if (in32) ldg256(src + r * ROW_BYTES, x[r]);
                    else ldg128x2(src + r * ROW_BYTES, x[r]);
                } else {
                    // the lane in which the column ends (or, shifted, begins or all but ends):
                    // through its place in the idle stage
                    const uint32_t count = n - e < EPL ? static_cast<uint32_t>(n - e) : EPL;
                    if constexpr (SHIFT)
                        load_end_unaligned(reinterpret_cast<const T*>(C.in) + e, count, reinterpret_cast<T*>(stage + lane * LANE_BYTES));
                    else
                        load_end(src + r * ROW_BYTES, count * static_cast<uint32_t>(sizeof(T)), stage_a + lane * LANE_BYTES);
#pragma unroll
                    for (uint32_t q = 0; q < 8; ++q) x[r][q] = lds32(stage_a + lane * LANE_BYTES + 4 * q);
                }
            }
        }
        const uint64_t ch = e0 >> p.chunk_log2;
        const uint64_t off0 = C.offsets[ch];
        const uint64_t blk = C.blk_base ? C.blk_base[ch >> (SCAN_BLOCK_LOG2 - p.chunk_log2)] : 0ull;
        it = next_item();
        if (it != NONE) load_mask(it);
        const uint64_t start = off0 + blk; // of the chunk
        const uint64_t off = start + before;

        uint32_t pos[ROWS];
        const uint32_t a = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(C.out) / sizeof(T) + off) % VEC);
        const uint32_t run = scan_item(bits, a, pos, lane);
        if (start > n || off + (run - a) > n) { // inconsistent offsets never write
            if (start != POISON && lane == 0) record_error(p.hdr, DEVERR_RANGE);
            continue;
        }
        write_item<T>(x, bits, pos, a, run,
                      C.out + (static_cast<int64_t>(off) - static_cast<int64_t>(a)) * static_cast<int64_t>(sizeof(T)), stage,
                      lut, lane);
    }

    if (!hybrid) return;
    // The items of sparse units. Those that pass 1 marked carry the mark of that pass's epoch, the one
    // before the current; without marks every item is tested. A warp looks at 32 work items at
    // a time, taken round robin over all warps so that marked items spread evenly.
    const uint32_t mark = p.item_flags ? epoch_mark(prev_epoch(*reinterpret_cast<const volatile uint32_t*>(&p.hdr->epoch))) : 0u;
    uint16_t* const list = reinterpret_cast<uint16_t*>(stage);
    const uint32_t split = p.num_sparse_items * 4 <= 2ull * total_warps ? 4u : 1u; // work items per 16K-element item
    const uint64_t num_work = p.num_sparse_items * split;
    for (uint64_t r0 = 0; warp_global + r0 * total_warps < num_work; r0 += 32) {
        const uint64_t mine = warp_global + (r0 + lane) * total_warps;
        const bool flagged = mine < num_work && (!p.item_flags || __ldg(p.item_flags + mine / split) == mark);
        uint32_t todo = __ballot_sync(0xffffffffu, flagged);
        while (todo) {
            const uint64_t work = warp_global + (r0 + (__ffs(todo) - 1)) * total_warps;
            todo &= todo - 1;
            const uint64_t item = work / split;
            const ColumnDesc& c = MULTI ? p.cols[__ldg(p.item_col + item)] : p.col0;
            const uint64_t e0 = (MULTI ? item + p.first_item - c.item_base : item) * 16384ull;
            if (split == 1u) sparse_groups<T, 4>(c, e0, p.chunk_log2, lane, list);
            else sparse_groups<T, 1>(c, e0 + (work & 3u) * 4096ull, p.chunk_log2, lane, list);
        }
    }
}

template <typename T, bool SHIFT>
cudaError_t launch_t(const WriteoutParams& p, uint32_t requested, int num_sms, cudaStream_t stream)
{
    const uint64_t items = p.num_units * (UNIT_TILES * TILE_BYTES / ITEM_BYTES);
    uint64_t blocks = (items + WARPS - 1) / WARPS;
    const uint64_t cap = requested ? requested : static_cast<uint64_t>(num_sms) * CTAS<T, SHIFT>; // one resident wave
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    WriteoutParams pp = p;
    const bool idle = sizeof(T) >= 4 && items >= 8 * blocks * WARPS;
    pp.throttle = !idle ? 0u : p.cols ? p.throttle : p.col0.d_count ? 1u : 0u;
    const dim3 g(static_cast<unsigned>(blocks)), b(WARPS * 32);
    cudaError_t e;
    const bool inside = (1u << p.chunk_log2) > ITEM_BYTES / sizeof(T); // items that start inside a chunk
    if (SHIFT && sizeof(T) > 1 && inside) e = launch_pdl(k_writeout_warp<T, false, SHIFT, (sizeof(T) > 1)>, g, b, 0, stream, pp);
    else if (SHIFT) e = launch_pdl(k_writeout_warp<T, false, SHIFT, false>, g, b, 0, stream, pp);
    else if (p.cols) e = launch_pdl(k_writeout_warp<T, true, false, false>, g, b, 0, stream, pp);
    else if (sizeof(T) > 1 && inside) e = launch_pdl(k_writeout_warp<T, false, false, (sizeof(T) > 1)>, g, b, 0, stream, pp);
    else e = launch_pdl(k_writeout_warp<T, false, false, false>, g, b, 0, stream, pp);
    note_launch();
    return e;
}

template <typename T>
cudaError_t launch_w(const WriteoutParams& p, uint32_t requested, int num_sms, cudaStream_t stream)
{
    const bool shift = !p.cols && (reinterpret_cast<uintptr_t>(p.col0.in) & 15u) != 0;
    return shift ? launch_t<T, true>(p, requested, num_sms, stream) : launch_t<T, false>(p, requested, num_sms, stream);
}

} // namespace

cudaError_t launch_writeout_warp(const WriteoutParams& p, uint32_t elem_bytes, uint32_t requested, int num_sms,
                                 cudaStream_t stream)
{
    switch (elem_bytes) {
        case 1: return launch_w<uint8_t>(p, requested, num_sms, stream);
        case 2: return launch_w<uint16_t>(p, requested, num_sms, stream);
        case 4: return launch_w<uint32_t>(p, requested, num_sms, stream);
        case 8: return launch_w<uint64_t>(p, requested, num_sms, stream);
        default: return cudaErrorInvalidValue;
    }
}

} // namespace cs
