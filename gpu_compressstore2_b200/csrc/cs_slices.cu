// cs_slices.cu — compaction in one kernel and one pass over HBM, for predicate compaction
// (compressstore_if: the selection is a comparison evaluated on the payload) and for the 1-pass form of
// the plain call (the selection is a mask in memory).
//
// The column is cut into slices of 32 KB: 8 warps x an item of 4 KB (cs_place.cuh). CTAs take slices
// in order from a device counter and work two slices ahead of themselves. In each turn a CTA
//   evaluates the slice two turns ahead: loads its mask, or its payload to compare, keeps the mask bits
//             in registers and publishes their count; a compared payload is dropped and stays in L2;
//   sums      the counts of the slices between its last one and the present one (about one per
//             CTA; published two turns ago, so it rarely waits): with the selected elements
//             before its last slice, which it carries along, that is the present slice's offset;
//   writes    the present slice: loads the payload (a comparison's again, now from L2), places and
//             stores the selected elements (an item with few is listed and gathered instead).
// The warps of a CTA meet at one barrier per turn. A CTA only ever waits for slices that running
// CTAs already hold, in order. Waits are bounded; a CTA that gives one up, or reads a total that no
// slice can have, records an error and writes nothing more, and the count reads CS_COUNT_ERROR. The epoch
// closes as soon as the last CTA has summed up for the last time, so nothing follows the writes (2^20
// u32: 7.1 -> 5.4 us).
//
// What bounds the predicate is the evaluation and the placing together, with a barrier per slice: half of the
// issue slots and half of DRAM at 24 warps per SM, the payload streaming at 4 to 5 TB/s. Per call on B200
// against a mask pass, pass 1 + 2 and the writeout, which read the payload from HBM twice, before ->
// now: 2^28 f32 x > c with 0.5 selected 459 -> 328 us, 0.01 259 -> 227, 0.1 414 -> 274, 0.9 556 -> 410;
// 2^27 f64 463 -> 313, 2^28 i16 289 -> 217, 2^28 u8 225 -> 179, 2^24 f32 41 -> 25, 2^20 18 -> 7.
// Tried: a look-back over slices instead of the carried sum (it grows with the number of slices: 494
// us at the best slice size), evaluating one slice ahead (365), slices of two items per warp
// (374 .. 384), 2 and 4 CTAs per SM (408, 378), the evaluated payload through shared memory by bulk
// copies (377). The 1-pass form's figures stand at slices_per_sm in cs_api.cu; what bounds it is the
// start (ticket, mask, payload one after another) for short columns and the barrier for long ones.
//
// A comparison of whole numbers is (x - lo) <= (hi - lo) in unsigned arithmetic, whatever the sign
// (the host turns each operator into bounds), one of floating numbers lo <= x && x <= hi; != is the
// negation of ==. Every ordered comparison with a NaN is false, != is true (C++ semantics).
//
// Reference: the reference evaluates the predicate on the host while packing the mask
// (gen_predicate, src/utils.cuh:102-122, with predicate_function x > threshold,
// src/main.cu:24-28,92) and copies mask and payload to the device before compacting.
#include <cstdint>
#include <cstring>
#include <type_traits>

#include <cuda_runtime.h>

#include "compressstore.h"
#include "cs_internal.cuh"
#include "cs_place.cuh"

namespace cs {

namespace {

constexpr uint32_t WARPS = 8;
constexpr uint32_t CTAS = 3; // per SM
// Selected elements of an item up to which they are listed and gathered (2^28 f32 with 0.01 selected
// 256 -> 227 us). Their ranks within a row take 8 bits.
constexpr uint32_t FEW = 64;
static_assert(FEW < 256, "ranks in 8 bits");

template <typename T>
__device__ __forceinline__ T from_bits(uint64_t b)
{
    T v;
    memcpy(&v, &b, sizeof(T)); // little-endian: the low bytes hold the value
    return v;
}

// Which bounds a comparison of floating numbers has (whole numbers take both in one).
enum Sides { FROM = 1, TO = 2, BOTH = 3, MASK = 4 }; // MASK: no comparison, the selection is a mask in memory

// Selected elements of a lane's 32 bytes, as bits.
template <typename T, int SIDES>
__device__ __forceinline__ uint32_t select_row(const uint32_t (&x)[8], T lo, T hi)
{
    constexpr uint32_t EPL = LANE_BYTES / sizeof(T);
    constexpr bool REAL = T(0.5) != T(0);
    uint32_t b = 0;
#pragma unroll
    for (uint32_t e = 0; e < EPL; ++e) {
        bool s;
        if constexpr (REAL) {
            T v;
            if constexpr (sizeof(T) == 8)
                v = __longlong_as_double(static_cast<long long>(static_cast<uint64_t>(x[2 * e]) | (static_cast<uint64_t>(x[2 * e + 1]) << 32)));
            else
                v = __uint_as_float(x[e]);
            s = SIDES == FROM ? lo <= v : SIDES == TO ? v <= hi : lo <= v && v <= hi;
        } else if constexpr (sizeof(T) == 8) {
            s = (static_cast<uint64_t>(x[2 * e]) | (static_cast<uint64_t>(x[2 * e + 1]) << 32)) - lo <= hi;
        } else {
            constexpr uint32_t PER = 4 / sizeof(T);
            s = static_cast<T>(static_cast<T>(x[e / PER] >> ((e % PER) * 8 * sizeof(T))) - lo) <= hi;
        }
        if (s) b |= 1u << e;
    }
    return b;
}

// T: uint8_t .. uint64_t (bounds lo and hi - lo), float, double (bounds lo, hi).
template <typename T, int SIDES>
__global__ void __launch_bounds__(WARPS * 32, CTAS) k_if(const SliceParams p)
{
    constexpr uint32_t EPL = LANE_BYTES / sizeof(T);
    constexpr uint32_t ROW = 32 * EPL;
    constexpr uint32_t ITEM = ROWS * ROW;
    constexpr uint32_t VEC = 16 / sizeof(T);
    constexpr bool MASKED = SIDES == MASK;
    constexpr int PK = EPL * ROWS > 32 ? EPL * ROWS / 32 : 1; // words that hold a lane's bits of an item
    constexpr uint32_t ROW_BITS = EPL == 32 ? 0xffffffffu : (1u << (EPL & 31u)) - 1u;
    __shared__ __align__(128) uint8_t s_stage[WARPS][STAGE_BYTES];
    __shared__ uint32_t s_lut[sizeof(T) == 1 ? PACK_TABLE_WORDS : 1];
    // By the slice's turn in this CTA (modulo 4: a slice is evaluated two turns ahead, one barrier
    // per turn), and the parts of a turn's sum by its parity.
    __shared__ uint32_t s_slice[4];                      // the slice of each turn
    __shared__ __align__(16) uint32_t s_total[4][WARPS]; // selected elements of each warp's part of it
    __shared__ uint32_t s_sum[4];                        // of the warps that have counted so far, and their number (bits 24 on)
    __shared__ __align__(16) uint32_t s_red[2][WARPS];   // parts of the sum of the totals since this CTA's last slice
    __shared__ uint32_t s_epoch, s_failed; // s_failed: what went wrong
    static_assert(WARPS == 8, "two vectors of warp totals");
    using U = typename std::conditional<sizeof(T) == 1, uint8_t, typename std::conditional<sizeof(T) == 2, uint16_t,
              typename std::conditional<sizeof(T) == 4, uint32_t, uint64_t>::type>::type>::type;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    uint8_t* const stage = s_stage[warp];
    const uint32_t stage_a = smem_u32(stage);
    const uint32_t lut = sizeof(T) == 1 ? smem_u32(s_lut) + lane * 4 : 0u;
    const T lo = from_bits<T>(p.lo), hi = from_bits<T>(p.hi);
    const uint32_t negate = p.negate ? ROW_BITS : 0u;
    const uint64_t n = p.n;
    const uint8_t* __restrict__ in = p.in;
    const bool in32 = (reinterpret_cast<uintptr_t>(in) & 31u) == 0;
    if constexpr (sizeof(T) == 1) fill_pack_table(s_lut, WARPS * 32);
    grid_dependency_wait();
    if (threadIdx.x == 0) {
        s_epoch = p.hdr->epoch;
        s_slice[0] = atomicAdd(&p.hdr->tile_counter, 1u);
        s_failed = 0u;
        for (uint32_t t = 0; t < 4; ++t) s_sum[t] = 0u;
    }
    __syncthreads();
    const uint32_t tag = slice_tag(s_epoch); // the epoch, but for two bits

    auto item_elem = [&](uint32_t slice) -> uint64_t { return (static_cast<uint64_t>(slice) * WARPS + warp) * ITEM; };
    // the lane's 32 bytes of row r of the item at e0, where the column ends in or before the item:
    // the lane in which it ends goes through its place in the idle stage
    auto load_ragged = [&](uint64_t e0, uint32_t r, uint32_t (&x)[8]) {
        const uint64_t e = e0 + r * ROW + lane * EPL;
        const uint8_t* src = in + e * sizeof(T);
        if (e + EPL <= n) {
            ldg128x2(src, x);
        } else if (e < n) {
            load_end(src, static_cast<uint32_t>(n - e) * static_cast<uint32_t>(sizeof(T)), stage_a + lane * LANE_BYTES);
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) x[q] = lds32(stage_a + lane * LANE_BYTES + 4 * q);
        }
    };
    auto load_whole = [&](const uint8_t* src, uint32_t (&x)[8]) {
        if (in32) ldg256(src, x);
        else ldg128x2(src, x);
    };
    auto row_bits = [&](const uint32_t (&b)[PK], uint32_t r) -> uint32_t {
        return (b[r * EPL / 32] >> (r * EPL % 32)) & ROW_BITS;
    };
    // this warp's part of a slice
    auto load_item = [&](uint32_t slice, uint32_t (&x)[ROWS][8]) {
        const uint64_t e0 = item_elem(slice);
        if (e0 + ITEM <= n) {
            const uint8_t* src = in + e0 * sizeof(T) + lane * LANE_BYTES;
#pragma unroll
            for (uint32_t r = 0; r < ROWS; ++r) load_whole(src + r * ROW_BYTES, x[r]);
        } else {
#pragma unroll
            for (uint32_t r = 0; r < ROWS; ++r) load_ragged(e0, r, x[r]);
        }
    };
    // the mask bits of this warp's part of a slice
    auto load_bits = [&](uint32_t slice, uint32_t (&m)[ROWS]) {
        const uint64_t e0 = item_elem(slice);
        const uint8_t* mb = reinterpret_cast<const uint8_t*>(p.mask_in);
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) {
            const uint64_t e = e0 + r * ROW + lane * EPL;
            uint32_t v = 0;
            if (e < n) {
                if constexpr (EPL == 32) v = __ldg(reinterpret_cast<const uint32_t*>(mb + (e >> 3)));
                else if constexpr (EPL == 16) v = __ldg(reinterpret_cast<const uint16_t*>(mb + (e >> 3)));
                else v = __ldg(mb + (e >> 3));
            }
            m[r] = v;
        }
    };
    // evaluates this warp's part of a slice into b; the last warp to do so publishes the slice's total
    auto evaluate = [&](uint32_t slice, const uint32_t (&m)[ROWS], const uint32_t (&x)[ROWS][8], uint32_t (&b)[PK], uint32_t turn) {
        const uint64_t e0 = item_elem(slice);
        const bool whole = e0 + ITEM <= n;
        uint32_t cnt = 0;
#pragma unroll
        for (int q = 0; q < PK; ++q) b[q] = 0;
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) {
            uint32_t s;
            if constexpr (!MASKED) s = select_row<T, SIDES>(x[r], lo, hi) ^ negate;
            else if constexpr (EPL == 4) s = (m[r] >> ((lane & 1u) * 4)) & 0xfu;
            else s = m[r];
            if (!whole) {
                const uint64_t e = e0 + r * ROW + lane * EPL;
                if (e + EPL > n) s = e < n ? s & ((1u << (n - e)) - 1u) : 0u; // n - e < EPL <= 32
            }
            b[r * EPL / 32] |= s << (r * EPL % 32);
        }
#pragma unroll
        for (int q = 0; q < PK; ++q) cnt += __popc(b[q]);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) {
            s_total[turn][warp] = cnt;
            const uint32_t before = atomicAdd(&s_sum[turn], cnt + (1u << 24));
            if (before >> 24 == WARPS - 1) {
                s_sum[turn] = 0u; // used again four turns on, past a barrier
                st_relaxed_gpu(&p.status[slice], slice_status(tag, (before & 0xffffffu) + cnt));
            }
        }
        if (!MASKED && p.mask) {
            // the lane's bits of the mask words that hold an element of the column
            const uint64_t bound = (n + 31) / 32 * 32;
#pragma unroll
            for (uint32_t r = 0; r < ROWS; ++r) {
                const uint64_t e = e0 + r * ROW + lane * EPL;
                uint8_t* mb = reinterpret_cast<uint8_t*>(p.mask) + (e >> 3);
                const uint32_t s = row_bits(b, r);
                if constexpr (EPL == 32) {
                    if (e < bound) *reinterpret_cast<uint32_t*>(mb) = s;
                } else if constexpr (EPL == 16) {
                    if (e < bound) *reinterpret_cast<uint16_t*>(mb) = static_cast<uint16_t>(s);
                } else if constexpr (EPL == 8) {
                    if (e < bound) *mb = static_cast<uint8_t>(s);
                } else {
                    const uint32_t pair = s | (__shfl_down_sync(0xffffffffu, s, 1) << 4);
                    if (e < bound && !(lane & 1u)) *mb = static_cast<uint8_t>(pair);
                }
            }
        }
    };
    uint32_t bits[PK], bits1[PK]; // of the slice to be written and the one after it
    uint64_t end = 0;  // selected elements before slice `done`
    uint32_t done = 0; // the slices up to this CTA's last one
    uint32_t turn = 0;
    // The first two slices, evaluated before any wait. A CTA takes each slice only when it is about to
    // evaluate it (or, in the loop, a turn before), so that the CTAs' slices interleave: a slice in front
    // of another CTA's is evaluated no later than that one.
#pragma unroll
    for (uint32_t t = 0; t < 2; ++t) {
        const uint32_t slice = s_slice[t];
        const bool some = slice < p.num_slices;
        if (some) {
            uint32_t x[ROWS][8], m[ROWS];
            if constexpr (MASKED) load_bits(slice, m);
            else load_item(slice, x);
            if (t == 0) evaluate(slice, m, x, bits, 0);
            else evaluate(slice, m, x, bits1, 1);
        }
        // (no second slice to ask for where every CTA has one)
        if (threadIdx.x == 0)
            s_slice[t + 1] = some && p.num_slices > gridDim.x ? atomicAdd(&p.hdr->tile_counter, 1u) : p.num_slices;
        __syncthreads();
    }
    // Thread 0 of every CTA, once its CTA has summed up for the last time: the last one to come closes the
    // epoch, and takes the count back if a wait gave up anywhere.
    auto leave = [&]() {
        // acquire: the other CTAs' mark and count, before the mark is read and the count replaced (a fence
        // here costs 0.4 us at 2^20 u32: it waits for this thread's own stores)
        if (atom_add_acquire_gpu(&p.hdr->done_counter, 1u) != gridDim.x - 1) return;
        volatile ws_header* vh = p.hdr;
        const uint32_t epoch = tag >> 2;
        if (vh->poison_epoch == epoch) *p.d_count = COUNT_ERROR;
        uint32_t following = epoch + 1u;
        if (following > EPOCH_MAX) {
            uint4* w = reinterpret_cast<uint4*>(p.hdr);
            for (uint64_t i = sizeof(ws_header) / 16u; i < vh->ws_bytes / 16u; ++i) w[i] = make_uint4(0, 0, 0, 0);
            vh->poison_epoch = vh->lost_epoch = 0u; // a new cycle must not meet an old one's marks
            following = EPOCH_MIN;
        }
        vh->tile_counter = 0u;
        vh->done_counter = 0u;
        vh->epoch = following;
    };
    if (threadIdx.x == 0 && s_slice[0] >= p.num_slices) leave();
    while (true) {
        const uint32_t slice = s_slice[turn];
        if (slice >= p.num_slices) break;
        const uint32_t later = (turn + 2) & 3u;
        const uint32_t next = s_slice[later]; // to be evaluated in this turn
        uint32_t ahead[PK];
        uint32_t x[ROWS][8];
        const bool more = next < p.num_slices;
        const uint64_t e0 = item_elem(slice);
        const uint32_t mine = s_total[turn][warp];
        const bool few = mine <= FEW;
        // This warp's item of the slice (of a comparison: from L2): few selected elements are listed and
        // gathered, otherwise the lanes with selected elements load theirs.
        auto load_selected = [&]() {
            if (few) return;
            if (e0 + ITEM <= n) {
                const uint8_t* src = in + e0 * sizeof(T) + lane * LANE_BYTES;
#pragma unroll
                for (uint32_t r = 0; r < ROWS; ++r)
                    if (row_bits(bits, r)) load_whole(src + r * ROW_BYTES, x[r]);
            } else {
#pragma unroll
                for (uint32_t r = 0; r < ROWS; ++r)
                    if (row_bits(bits, r)) load_ragged(e0, r, x[r]);
            }
        };
        if constexpr (MASKED) load_selected();
        uint32_t m[ROWS];
        if (more) {
            if constexpr (MASKED) load_bits(next, m);
            else load_item(next, x);
        }
        if (threadIdx.x == 0) s_slice[(turn + 3) & 3u] = more ? atomicAdd(&p.hdr->tile_counter, 1u) : next;
        // the totals of the slices since this CTA's last one, 512 at a time
        uint32_t* const red = s_red[turn & 1u];
        for (; slice - done > 2 * WARPS * 32; done += 2 * WARPS * 32) {
            const uint32_t wrong = poll_totals<WARPS * 32, WARPS * ITEM>(p.status, done, done + 2 * WARPS * 32, tag, p.timeout_ns, red);
            if (wrong) s_failed = wrong;
            __syncthreads();
#pragma unroll
            for (uint32_t w = 0; w < WARPS; ++w) end += red[w];
            __syncthreads();
        }
        const uint32_t wrong = poll_totals<WARPS * 32, WARPS * ITEM>(p.status, done, slice, tag, s_failed ? 0ull : p.timeout_ns, red);
        if (wrong) s_failed = wrong;
        if (more) evaluate(next, m, x, ahead, later);
        if constexpr (!MASKED) load_selected();
        __syncthreads(); // the sums of this turn; every warp has left the turn before
        const uint4 t0 = lds128(s_total[turn]), t1 = lds128(s_total[turn] + 4);
        const uint4 r0 = lds128(red), r1 = lds128(red + 4);
        const uint64_t base = end + (static_cast<uint64_t>(r0.x) + r0.y + r0.z + r0.w) + (static_cast<uint64_t>(r1.x) + r1.y + r1.z + r1.w);
        end = base + (t0.x + t0.y + t0.z + t0.w + t1.x + t1.y + t1.z + t1.w);
        done = slice + 1;
        const bool failed = s_failed != 0u;
        if (threadIdx.x == 0) {
            if (failed) {
                record_error(p.hdr, s_failed);
                reinterpret_cast<volatile ws_header*>(p.hdr)->poison_epoch = tag >> 2;
            }
            if (slice == p.num_slices - 1) *p.d_count = end;
            if (s_slice[(turn + 1) & 3u] >= p.num_slices) { // the CTA's last slice
                if (failed || slice == p.num_slices - 1) __threadfence(); // the mark, the count before `leave`
                leave();
            }
        }
        if (!failed && mine != 0u) {
            const uint64_t off = base + (warp > 0 ? t0.x : 0u) + (warp > 1 ? t0.y : 0u) + (warp > 2 ? t0.z : 0u) + (warp > 3 ? t0.w : 0u) +
                                 (warp > 4 ? t1.x : 0u) + (warp > 5 ? t1.y : 0u) + (warp > 6 ? t1.z : 0u);
            if (few) {
                uint16_t* const list = reinterpret_cast<uint16_t*>(stage);
                // ranks row by row: at most FEW elements, so the four rows' counts fit one scanned word
                uint32_t own = 0;
#pragma unroll
                for (uint32_t r = 0; r < ROWS; ++r) own |= static_cast<uint32_t>(__popc(row_bits(bits, r))) << (8 * r);
                const uint32_t incl = warp_incl_scan(own, lane);
                const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
                const uint32_t excl = incl - own;
                uint32_t before = 0;
#pragma unroll
                for (uint32_t r = 0; r < ROWS; ++r) {
                    uint32_t at = before + ((excl >> (8 * r)) & 0xffu);
                    for (uint32_t m = row_bits(bits, r); m != 0u; m &= m - 1)
                        list[at++] = static_cast<uint16_t>(r * ROW + lane * EPL + __ffs(m) - 1);
                    before += (all >> (8 * r)) & 0xffu;
                }
                __syncwarp();
                const U* src = reinterpret_cast<const U*>(in) + e0;
                U* dst = reinterpret_cast<U*>(p.out) + off;
                for (uint32_t j = lane; j < mine; j += 32) dst[j] = ldg_gather(src + list[j]);
                __syncwarp();
            } else {
                const uint32_t a = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(p.out) / sizeof(T) + off) % VEC);
                uint32_t rb[ROWS], pos[ROWS];
#pragma unroll
                for (uint32_t r = 0; r < ROWS; ++r) rb[r] = row_bits(bits, r);
                const uint32_t run = scan_item(rb, a, pos, lane);
                write_item<U>(x, rb, pos, a, run,
                              p.out + (static_cast<int64_t>(off) - static_cast<int64_t>(a)) * static_cast<int64_t>(sizeof(T)),
                              stage, lut, lane);
            }
        }
        turn = (turn + 1) & 3u;
#pragma unroll
        for (int q = 0; q < PK; ++q) {
            bits[q] = bits1[q];
            bits1[q] = ahead[q];
        }
    }
}

template <typename T, int SIDES>
cudaError_t launch_s(const SliceParams& p, int num_sms, cudaStream_t stream)
{
    SliceParams q = p;
    q.num_slices = static_cast<uint32_t>(slices_of(p.n, sizeof(T)));
    uint64_t grid = p.grid ? p.grid : static_cast<uint64_t>(num_sms) * CTAS;
    if (grid > q.num_slices) grid = q.num_slices;
    return launch_pdl(k_if<T, SIDES>, dim3(static_cast<unsigned>(grid)), dim3(WARPS * 32), 0, stream, q);
}

template <typename T>
cudaError_t launch_t(const SliceParams& p, int num_sms, cudaStream_t stream)
{
    if (p.mask_in) return launch_s<T, MASK>(p, num_sms, stream);
    return launch_s<T, BOTH>(p, num_sms, stream);
}

template <typename T>
cudaError_t launch_real(const SliceParams& p, int num_sms, cudaStream_t stream)
{
    if (p.sides == FROM) return launch_s<T, FROM>(p, num_sms, stream);
    if (p.sides == TO) return launch_s<T, TO>(p, num_sms, stream);
    return launch_s<T, BOTH>(p, num_sms, stream);
}

} // namespace

uint64_t slices_of(uint64_t n, uint32_t elem_bytes)
{
    const uint64_t items = (n * elem_bytes + ITEM_BYTES - 1) / ITEM_BYTES;
    return (items + WARPS - 1) / WARPS;
}

cudaError_t launch_if(const SliceParams& p, int type, int num_sms, cudaStream_t stream)
{
    cudaError_t e;
    switch (type) {
        case CS_U8:
        case CS_I8: e = launch_t<uint8_t>(p, num_sms, stream); break;
        case CS_U16:
        case CS_I16: e = launch_t<uint16_t>(p, num_sms, stream); break;
        case CS_U32:
        case CS_I32: e = launch_t<uint32_t>(p, num_sms, stream); break;
        case CS_U64:
        case CS_I64: e = launch_t<uint64_t>(p, num_sms, stream); break;
        case CS_F32: e = launch_real<float>(p, num_sms, stream); break;
        case CS_F64: e = launch_real<double>(p, num_sms, stream); break;
        default: return cudaErrorInvalidValue;
    }
    note_launch();
    return e;
}

cudaError_t launch_onepass(const SliceParams& p, uint32_t elem_bytes, int num_sms, cudaStream_t stream)
{
    cudaError_t e;
    switch (elem_bytes) {
        case 1: e = launch_t<uint8_t>(p, num_sms, stream); break;
        case 2: e = launch_t<uint16_t>(p, num_sms, stream); break;
        case 4: e = launch_t<uint32_t>(p, num_sms, stream); break;
        case 8: e = launch_t<uint64_t>(p, num_sms, stream); break;
        default: return cudaErrorInvalidValue;
    }
    note_launch();
    return e;
}

} // namespace cs
