// cs_place.cuh — a warp's item: 4 KB of payload held in registers, its selected elements put in
// order into a stage of the warp in shared memory, and the stage written out. Used by the 3-pass
// writeout (cs_writeout.cu), the slices (cs_slices.cu) and the pattern compaction (cs_pattern.cu).
#pragma once
#include <cstdint>

#include "cs_ptx.cuh"

namespace cs {

constexpr uint32_t ROWS = 4;                              // 32-byte loads per lane and item
constexpr uint32_t LANE_BYTES = 32;                       // payload bytes per lane and row
constexpr uint32_t ROW_BYTES = 32 * LANE_BYTES;
constexpr uint32_t ITEM_BYTES = ROWS * ROW_BYTES;         // 4 KB
constexpr uint32_t STAGE_BYTES = ITEM_BYTES + 128;        // selected elements from any 16-byte phase, whole lines

__device__ __forceinline__ void ldg256(const void* p, uint32_t (&x)[8])
{
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                 : "l"(p));
}

__device__ __forceinline__ void ldg128x2(const void* p, uint32_t (&x)[8])
{
    const uint4 a = __ldg(static_cast<const uint4*>(p)), b = __ldg(static_cast<const uint4*>(p) + 1);
    x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
    x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
}

// Where byte `a` of a stage lies: its 16-byte slots change places within their 128-byte line by the
// line's number (m = 0x70; 0: they do not). Elements that the lanes of a warp store at strides of 8
// words and its multiples (runs of selected elements: a lane holds 32 bytes) otherwise meet in
// few banks.
__device__ __forceinline__ uint32_t stage_swizzle(uint32_t a, uint32_t m)
{
    return a ^ ((a >> 3) & m);
}

__device__ __forceinline__ void sts32(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t lo, uint32_t hi)
{
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(lo), "r"(hi) : "memory");
}
__device__ __forceinline__ void sts8(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(static_cast<uint16_t>(v)) : "memory");
}
__device__ __forceinline__ uint4 lds128_at(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// What a lane's run of 1-byte elements leaves past its last whole word: `f8` bits of acc, of
// which the lowest lo8 are earlier lanes'.
struct Tail {
    uint32_t acc, at, f8, lo8;
};

// One lane's row (32 payload bytes in x, `bits` selecting from them) to the stage address `at`.
// SWZ: through stage_swizzle (never for 1-byte elements, whose words spread by themselves).
template <typename T, bool SWZ>
__device__ __forceinline__ Tail place_row(const uint32_t (&x)[8], uint32_t bits, uint32_t at, uint32_t lut)
{
    constexpr uint32_t M = SWZ ? 0x70u : 0u;
    Tail t{0u, at, 0u, 0u};
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e)
            if ((bits >> e) & 1u) {
                sts64(stage_swizzle(at, M), x[2 * e], x[2 * e + 1]);
                at += 8;
            }
    } else if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e)
            if ((bits >> e) & 1u) {
                sts32(stage_swizzle(at, M), x[e]);
                at += 4;
            }
    } else if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (uint32_t e = 0; e < 16; ++e)
            if ((bits >> e) & 1u) {
                sts16(stage_swizzle(at, M), e & 1u ? x[e / 2] >> 16 : x[e / 2]);
                at += 2;
            }
    } else {
        // `fill`: bits placed so far, from the start of the run's first word; a word is complete
        // when bit 5 of it changes (shifts take it modulo 32)
        uint32_t fill = at * 8u;
        const uint32_t word0 = fill >> 5;
        t.lo8 = fill & 31u;
        at &= ~3u;
        uint32_t acc = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            // the table's entry of 4 mask bits: byte selectors that pack the selected bytes (low
            // 16 bits; 4 selects a zero), 8 x their number (high 16 bits)
            const uint32_t ent = lds32(lut + ((k < 2 ? bits << (7 - 4 * k) : bits >> (4 * k - 7)) & 0x780u));
            const uint32_t pk = __byte_perm(x[k], 0u, ent);
            const uint32_t next = fill + (ent >> 16);
            const uint32_t w0 = acc | __funnelshift_l(0u, pk, fill);
            const uint32_t w1 = __funnelshift_l(pk, 0u, fill);
            if ((next ^ fill) & 32u) {
                sts32(at, w0);
                at += 4;
                acc = w1;
            } else {
                acc = w0;
            }
            fill = next;
        }
        if ((fill >> 5) != word0) t.lo8 = 0;
        t.acc = acc;
        t.at = at;
        t.f8 = fill & 31u;
    }
    return t;
}

__device__ __forceinline__ void place_tail(const Tail& t)
{
#pragma unroll
    for (uint32_t b = 0; b < 3; ++b)
        if (b * 8 >= t.lo8 && b * 8 < t.f8) sts8(t.at + b, t.acc >> (8 * b));
}

// The table that place_row reads for 1-byte elements: one copy per lane of the 16 entries, so its
// reads do not conflict. Called by all `threads` threads; a barrier before its use.
constexpr uint32_t PACK_TABLE_WORDS = 16 * 32;
__device__ __forceinline__ void fill_pack_table(uint32_t* table, uint32_t threads)
{
    for (uint32_t i = threadIdx.x; i < PACK_TABLE_WORDS; i += threads) {
        const uint32_t nib = i >> 5;
        uint32_t sel = 0x4444u, k = 0;
        for (uint32_t b = 0; b < 4; ++b)
            if ((nib >> b) & 1u) {
                sel = (sel & ~(0xfu << (4 * k))) | (b << (4 * k));
                ++k;
            }
        table[i] = sel | (k << 19);
    }
}

// The end of a column, `bytes` < LANE_BYTES from `src` (16-byte aligned) to `tmp` in shared memory, by one
// lane: both halves go out together and hold no registers (elements one after another through a loop: 1-pass
// calls of 3 x 10^6 u8 6.97 -> 5.89 us).
__device__ __forceinline__ void load_end(const uint8_t* src, uint32_t bytes, uint32_t tmp)
{
    const uint32_t first = bytes < 16u ? bytes : 16u;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tmp), "l"(src), "r"(first) : "memory");
    if (bytes > 16u)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tmp + 16u), "l"(src + 16), "r"(bytes - 16u) : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The same for an element-aligned `in` and up to LANE_BYTES, eight elements at a time.
template <typename T>
__device__ __forceinline__ void load_end_unaligned(const T* __restrict__ in, uint32_t count, T* tmp)
{
    constexpr uint32_t BATCH = LANE_BYTES / sizeof(T) < 8 ? LANE_BYTES / sizeof(T) : 8;
    for (uint32_t i = 0; i < count; i += BATCH) {
        T v[BATCH];
#pragma unroll
        for (uint32_t k = 0; k < BATCH; ++k)
            if (i + k < count) v[k] = __ldg(in + i + k);
#pragma unroll
        for (uint32_t k = 0; k < BATCH; ++k)
            if (i + k < count) tmp[i + k] = v[k];
    }
}

// Elements [a, run) of the stage (placed with swizzle m) to gdst + the same positions (gdst 16-byte
// aligned, a within its first vector): whole 16-byte vectors, and the ragged ends element by
// element (lanes 0-15 the head, lanes 16-31 the tail).
template <typename T>
__device__ __forceinline__ void emit_stage(uint8_t* gdst, const uint8_t* stage, uint32_t a, uint32_t run, uint32_t lane,
                                           uint32_t m)
{
    constexpr uint32_t VEC = 16 / sizeof(T);
    const uint32_t base = smem_u32(stage);
    const uint32_t v0 = a ? 1u : 0u, v1 = run / VEC;
    for (uint32_t v = v0 + lane; v < v1; v += 32) stg128_cs(gdst + v * 16u, lds128_at(stage_swizzle(base + v * 16u, m)));
    const uint32_t i = lane & 15u;
    if (i < VEC) {
        const uint32_t e = lane & 16u ? v1 * VEC + i : i;
        const bool st = lane & 16u ? v1 >= v0 && e < run : a != 0u && e >= a && e < run;
        if (st) {
            const uint32_t at = stage_swizzle(base + e * static_cast<uint32_t>(sizeof(T)), m) - base;
            reinterpret_cast<T*>(gdst)[e] = *reinterpret_cast<const T*>(stage + at);
        }
    }
}

// Stage positions of a lane's four runs, from the lanes' counts: two rows (at most 1024 elements
// each) per packed scan. `a`: position of the item's first selected element; returns the end.
__device__ __forceinline__ uint32_t scan_item(const uint32_t (&bits)[ROWS], uint32_t a, uint32_t (&pos)[ROWS], uint32_t lane)
{
    uint32_t run = a;
#pragma unroll
    for (uint32_t r = 0; r < ROWS; r += 2) {
        const uint32_t own = __popc(bits[r]) | (__popc(bits[r + 1]) << 16);
        const uint32_t incl = warp_incl_scan(own, lane);
        const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
        pos[r] = run + ((incl - own) & 0xffffu);
        run += all & 0xffffu;
        pos[r + 1] = run + ((incl - own) >> 16);
        run += all >> 16;
    }
    return run;
}

// The selected elements of an item (bits of x) through the stage to gdst + [a, run): the positions
// are scan_item's, gdst is 16-byte aligned.
template <typename T>
__device__ __forceinline__ void write_item(const uint32_t (&x)[ROWS][8], const uint32_t (&bits)[ROWS],
                                           const uint32_t (&pos)[ROWS], uint32_t a, uint32_t run, uint8_t* gdst,
                                           uint8_t* stage, uint32_t lut, uint32_t lane)
{
    constexpr uint32_t ITEM = ITEM_BYTES / sizeof(T);
    const uint32_t base = smem_u32(stage);
    uint32_t swz = 0u;
    Tail tail[ROWS];
    __syncwarp(); // lanes that passed their payload through the stage have read it
    if ((sizeof(T) == 2 || sizeof(T) == 4) && run - a > ITEM / 16 * 15) {
        // nearly all of the item is selected: the lanes' elements lie 8 words apart (2^28 u32 runs of
        // 4096 262 -> 239 us, 2^28 u16 205 -> 170, p = 0.99 247 -> 204; with every item 2^28 u16
        // p = 0.5 151 -> 162)
        swz = 0x70u;
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r)
            place_row<T, (sizeof(T) > 1)>(x[r], bits[r], base + pos[r] * static_cast<uint32_t>(sizeof(T)), lut);
    } else {
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r)
            tail[r] = place_row<T, false>(x[r], bits[r], base + pos[r] * static_cast<uint32_t>(sizeof(T)), lut);
    }
    if constexpr (sizeof(T) == 1) {
        __syncwarp(); // every whole word is in the stage before the partial ones
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) place_tail(tail[r]);
    }
    __syncwarp();
    emit_stage<T>(gdst, stage, a, run, lane, swz);
    __syncwarp(); // the stage is rewritten by the next item
}

} // namespace cs
