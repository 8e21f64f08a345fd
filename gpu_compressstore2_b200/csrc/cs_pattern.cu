// cs_pattern.cu — compaction by a periodic pattern instead of a mask in memory.
//
// Element i is selected when bit (i % L) of `pattern` is set (LSB-first, 1 <= L <= 32). With
// P = popcount of the pattern's L bits, output j is input (j / P) * L + pos[j % P], pos[r]
// being the r-th set bit: every output has a closed-form source, so there is no popcount
// pass, no scan and no mask read. Three kernels:
//
// k_pattern gathers. A warp produces runs of 128 output bytes (256 for 8-byte elements): each
// lane 4 consecutive bytes of them (1, 2 or 4 elements) or one 8-byte element, so that one load
// instruction of the warp falls on the few lines that its outputs come from and one store
// instruction writes whole lines. The offsets of a lane's sources repeat every P such runs: they
// come from a table in shared memory, and a thread divides twice. A thread keeps the loads of
// PATTERN_RUNS runs in flight before it stores. Where the selected elements lie 64 bytes and more
// apart a load fetches 64 bytes instead of a line (2^28 u32, 1 of 32: 163 -> 91 us).
//
// k_pattern_dense streams the input through registers and a stage per warp as the 3-pass
// writeout does (cs_writeout.cu), with mask bits and positions from the pattern; it runs at the HBM
// rate from about a third selected on (2^28 u32, 31 of 32: 2.11 GB in 322 us).
//
// k_pattern_all copies where everything is selected.
// Reference: bench9_pattern (src/benchmarks.cuh:397-416) over launch_pattern_proc /
// kernel_pattern_proc (src/kernels/kernel_pattern.cuh:13-131), whose pattern is read from
// the most significant bit (element i <-> bit 31 - i % L); pass __brev of such a pattern.
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "compressstore.h"
#include "cs_internal.cuh"
#include "cs_place.cuh"

namespace cs {

namespace {

constexpr uint32_t PATTERN_RUNS = 8;
// CTAs per SM. 5 or 6 are resident; 4- and 8-byte elements keep the memory busier with a second set of blocks
// that start as the first end (8 / 16, us, output not 16-byte aligned: 2^28 u32 1 of 2 278 / 250, 2 of 3 342 / 288, 2^26
// u64 6 of 7 172 / 161), where 2-byte ones lose (2^28 1 of 2 179 / 194) and bytes do not care (8 of 8 269 / 262, 2 of 3 6.2 / 6.2).
template <typename T> constexpr uint32_t PATTERN_CTAS = sizeof(T) >= 4 ? 16u : 8u;

// VEC_OUT: the output is aligned to a lane's bytes. APART: the selected elements lie 64 bytes and
// more apart on average, so a load fetches 64 bytes rather than a line.
template <typename T, bool VEC_OUT, bool APART>
__global__ void __launch_bounds__(256) k_pattern(const T* __restrict__ in, T* __restrict__ out, uint32_t pattern,
                                                 uint32_t L, uint32_t P, uint64_t count, uint64_t* d_count)
{
    constexpr uint32_t G = sizeof(T) < 4 ? 4 / sizeof(T) : 1; // elements per lane and run
    constexpr uint32_t RUN = 32 * G;                          // outputs per run
    constexpr uint32_t U = PATTERN_RUNS;
    __shared__ uint32_t s_pos[32];
    // source offset of output i of P consecutive runs, from the period the first one starts
    __shared__ __align__(8) uint16_t s_off[RUN * 32];
    if (threadIdx.x < 32) {
        const uint32_t b = threadIdx.x;
        if (b < L && ((pattern >> b) & 1u)) s_pos[__popc(pattern & ((1u << b) - 1u))] = b;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_count = count;
    __syncthreads();
    // (one division; the table of a dense pattern is long, and a short column has time for little else)
    uint32_t tq = threadIdx.x / P, tr = threadIdx.x % P;
    const uint32_t tdq = 256 / P, tdr = 256 % P;
    for (uint32_t i = threadIdx.x; i < RUN * P; i += 256) {
        s_off[i] = static_cast<uint16_t>(tq * L + s_pos[tr]);
        tq += tdq;
        tr += tdr;
        if (tr >= P) {
            tr -= P;
            ++tq;
        }
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    // Numbers of warps of a bounded grid: divided in 32 bits, which a short column notices (2^20 u64, 6 of 7, 6.1 -> 4.7 us).
    // The loop of 2-byte elements that are stored one by one comes out better from 64 (2^28, us, 32 / 64: 1 of 2 196 /
    // 179, 2 of 3 256 / 230, 8 of 8 372 / 328).
    using Index = std::conditional_t<sizeof(T) == 2 && !VEC_OUT, uint64_t, uint32_t>;
    const Index s_first = ((static_cast<Index>(blockIdx.x) * 256u + threadIdx.x) >> 5) * U;
    const Index step = static_cast<Index>(gridDim.x) * 8u * U; // runs between a warp's groups
    const uint64_t runs = (count + RUN - 1) / RUN;
    const Index dq = step / P;
    const uint32_t dr = static_cast<uint32_t>(step % P);
    const uint32_t period = RUN * L; // inputs of P runs
    uint64_t q = s_first / P;
    uint32_t r = static_cast<uint32_t>(s_first % P);
    for (uint64_t s0 = s_first; s0 < runs; s0 += step) {
        T x[U][G];
        const T* src = in + q * period;
        uint32_t rk = r;
        const uint64_t j0 = s0 * RUN + lane * G; // this lane's first output
        const bool whole = (s0 + U) * RUN <= count;
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            uint16_t off[G];
            if constexpr (G == 4) *reinterpret_cast<uint2*>(off) = *reinterpret_cast<const uint2*>(&s_off[rk * RUN + lane * G]);
            else if constexpr (G == 2) *reinterpret_cast<uint32_t*>(off) = *reinterpret_cast<const uint32_t*>(&s_off[rk * RUN + lane * G]);
            else off[0] = s_off[rk * RUN + lane];
#pragma unroll
            for (uint32_t e = 0; e < G; ++e)
                if (whole || j0 + u * RUN + e < count) x[u][e] = APART ? ldg_gather(src + off[e]) : __ldg(src + off[e]);
            if (++rk == P) {
                rk = 0;
                src += period;
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            T* dst = out + j0 + u * RUN;
            if (VEC_OUT && G > 1 && (whole || j0 + u * RUN + G <= count)) {
                uint32_t v;
                if constexpr (G == 4) v = x[u][0] | x[u][1 % G] << 8 | x[u][2 % G] << 16 | static_cast<uint32_t>(x[u][3 % G]) << 24;
                else v = static_cast<uint32_t>(x[u][0]) | static_cast<uint32_t>(x[u][1 % G]) << 16;
                __stcs(reinterpret_cast<uint32_t*>(dst), v);
            } else {
#pragma unroll
                for (uint32_t e = 0; e < G; ++e)
                    if (whole || j0 + u * RUN + e < count) __stcs(dst + e, x[u][e]);
            }
        }
        q += dq;
        r += dr;
        if (r >= P) {
            r -= P;
            ++q;
        }
    }
}

// A pattern that selects everything: the column, 16 bytes at a time where it lies so (all pointers 16-byte
// aligned), and what is left of it byte by byte. 2^28 u16 171 us, 1 byte 88 (the dense kernel 312 and 109).
constexpr uint32_t COPY_CTAS = 2; // per SM (1 GB of 8-byte elements: 2 172 us, 3 180, 4 180, 8 177)
__global__ void __launch_bounds__(256) k_pattern_all(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t bytes,
                                                     uint64_t count, uint64_t* d_count)
{
    constexpr uint32_t U = 4;
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_count = count;
    const uint64_t vectors = bytes / 16;
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * 256 * U;
    const uint4* __restrict__ src = reinterpret_cast<const uint4*>(in);
    uint4* __restrict__ dst = reinterpret_cast<uint4*>(out);
    for (uint64_t v0 = static_cast<uint64_t>(blockIdx.x) * 256 * U + threadIdx.x; v0 < vectors; v0 += step) {
        uint4 x[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
            if (v0 + u * 256 < vectors) x[u] = __ldg(src + v0 + u * 256);
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
            if (v0 + u * 256 < vectors) __stcs(dst + v0 + u * 256, x[u]);
    }
    const uint32_t rest = static_cast<uint32_t>(bytes % 16);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x < rest) out[vectors * 16 + threadIdx.x] = in[vectors * 16 + threadIdx.x];
}

// Dense patterns: items of 4 KB of payload per warp as in the 3-pass writeout (cs_writeout.cu),
// with the mask bits and the positions from the pattern instead of a mask and a scan: element e
// has rank (e / L) * P + the pattern's set bits below e % L. `rep`: the pattern repeated over 64
// bits. The input 16-byte aligned.
constexpr uint32_t DENSE_WARPS = 8;
constexpr uint32_t DENSE_CTAS = 3;

template <typename T, bool SWZ>
__global__ void __launch_bounds__(DENSE_WARPS * 32, DENSE_CTAS)
    k_pattern_dense(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t n, uint32_t pattern, uint64_t rep,
                    uint32_t L, uint32_t P, uint64_t count, uint64_t* d_count)
{
    constexpr uint32_t EPL = LANE_BYTES / sizeof(T);
    constexpr uint32_t ROW = 32 * EPL;
    constexpr uint32_t ITEM = ROWS * ROW;
    constexpr uint32_t VEC = 16 / sizeof(T);
    constexpr uint32_t BITS = EPL == 32 ? 0xffffffffu : (1u << (EPL & 31u)) - 1u;
    __shared__ __align__(128) uint8_t s_stage[DENSE_WARPS][STAGE_BYTES];
    __shared__ uint32_t s_lut[sizeof(T) == 1 ? PACK_TABLE_WORDS : 1];
    if constexpr (sizeof(T) == 1) {
        fill_pack_table(s_lut, DENSE_WARPS * 32);
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) *d_count = count;
    uint8_t* const stage = s_stage[warp];
    const uint32_t stage_a = smem_u32(stage);
    const uint32_t lut = sizeof(T) == 1 ? smem_u32(s_lut) + lane * 4 : 0u;
    const bool in32 = (reinterpret_cast<uintptr_t>(in) & 31u) == 0;
    const uint32_t step = gridDim.x * DENSE_WARPS * ITEM; // of a resident grid: both in 32 bits
    const uint32_t first = (blockIdx.x * DENSE_WARPS + warp) * ITEM;
    uint64_t e0 = first;
    // the period and the place within it of this lane's first element; both advance without
    // further divisions
    const uint32_t dq = step / L, dr = step % L;
    uint64_t q = (first + lane * EPL) / L;
    uint32_t r = (first + lane * EPL) % L;
    const uint32_t row_q = ROW / L, row_r = ROW % L;
    for (; e0 < n; e0 += step) {
        const bool whole = e0 + ITEM <= n;
        const uint8_t* src = in + e0 * sizeof(T) + lane * LANE_BYTES;
        uint32_t bits[ROWS], rank[ROWS], x[ROWS][8];
        uint32_t rk = r, qk = static_cast<uint32_t>(q); // ranks within an item fit 32 bits
#pragma unroll
        for (uint32_t k = 0; k < ROWS; ++k) {
            uint32_t b = __funnelshift_r(static_cast<uint32_t>(rep), static_cast<uint32_t>(rep >> 32), rk) & BITS;
            const uint64_t e = e0 + k * ROW + lane * EPL;
            if (!whole && e + EPL > n) b &= e < n ? (1u << (n - e)) - 1u : 0u;
            bits[k] = b;
            rank[k] = qk * P + __popc(pattern & ((1u << rk) - 1u));
            if (b) {
                if (whole || e + EPL <= n) {
                    if (in32) ldg256(src + k * ROW_BYTES, x[k]);
                    else ldg128x2(src + k * ROW_BYTES, x[k]);
                } else {
                    // the lane in which the column ends: through the idle stage
                    load_end(src + k * ROW_BYTES, static_cast<uint32_t>(n - e) * static_cast<uint32_t>(sizeof(T)), stage_a + lane * LANE_BYTES);
#pragma unroll
                    for (uint32_t w = 0; w < 8; ++w) x[k][w] = lds32(stage_a + lane * LANE_BYTES + 4 * w);
                }
            }
            qk += row_q;
            rk += row_r;
            if (rk >= L) {
                rk -= L;
                ++qk;
            }
        }
        const uint64_t off = __shfl_sync(0xffffffffu, q * P + __popc(pattern & ((1u << r) - 1u)), 0); // rank of e0
        const uint32_t a = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(out) / sizeof(T) + off) % VEC);
        const uint32_t end = __shfl_sync(0xffffffffu, rank[ROWS - 1] + __popc(bits[ROWS - 1]), 31);
        const uint32_t run = a + (whole ? end - static_cast<uint32_t>(off) : static_cast<uint32_t>(count - off));
        __syncwarp(); // the ragged lane has read its place in the stage
        Tail tail[ROWS];
#pragma unroll
        for (uint32_t k = 0; k < ROWS; ++k)
            tail[k] = place_row<T, SWZ>(x[k], bits[k],
                                        stage_a + (rank[k] - static_cast<uint32_t>(off) + a) * static_cast<uint32_t>(sizeof(T)), lut);
        if constexpr (sizeof(T) == 1) {
            __syncwarp(); // every whole word is in the stage before the partial ones
#pragma unroll
            for (uint32_t k = 0; k < ROWS; ++k) place_tail(tail[k]);
        }
        __syncwarp();
        emit_stage<T>(out + (static_cast<int64_t>(off) - static_cast<int64_t>(a)) * static_cast<int64_t>(sizeof(T)), stage, a,
                      run, lane, SWZ ? 0x70u : 0u);
        __syncwarp(); // the stage is rewritten by the next item
        q += dq;
        r += dr;
        if (r >= L) {
            r -= L;
            ++q;
        }
    }
}

// Which kernel a pattern takes. The gather's time follows the outputs, the dense kernel's the inputs.
// Per call on B200, n = 2^28 (2^27 for 8 bytes), gather / dense, us, by selected share P / L:
//           0.25       0.33       0.375      0.43       0.5        0.75       0.97
//   1 byte  67 / 75    - / 78     108 / 76   119 / 80   136 / 78   - / 80     257 / 88
//   2       105 / 110  120 / 147  147 / 118  162 / 131  175 / 145  - / 159    333 / 172
//   4       201 / 202  214 / 230  233 / 217  250 / 230  266 / 245  318 / 288  371 / 322
//   8       196 / 196  209 / 214  230 / 215  241 / 230  252 / 242  306 / 282  349 / 325
// (dense at the better of 2 and 3 CTAs per SM; one thread per 16 output bytes, which both replace:
// 1 byte 131 .. 156 .. 297, 2 bytes 158 .. 164 .. 318, 4 bytes 213 .. 256 .. 438).
//
// Short columns are gathered whatever the share: the dense kernel starts more slowly. Gather / dense, us, by
// bytes of payload (4.1 is what the launches themselves take): 1 byte, 4 of 8, 1 MB 4.1 / 6.1, 2 MB 4.4 / 6.2, 4 MB
// 6.2 / 6.2; 2 bytes, 6 of 7, 1 MB 4.1 / 6.2, 2 MB 5.2 / 6.2, 2 of 3, 2 MB 4.2 / 4.2; 4 bytes 2 MB 4.0 / 4.2. 8 bytes stay
// with it longer: 4 of 8, 32 MB 14.2 / 14.2, 64 MB 19.1 / 20.4, but 6 of 7, 64 MB 24.6 / 23.5, 512 MB 167 / 166.
// And so are halves in runs of 32 bytes and more, of which the gather reads whole sectors and has nothing to
// pack: 8 bytes, 16 of 32 in one run, 2^26 94 / 111, 2^24 27 / 32; 4 bytes 65.7 / 72 at 2^26, 262 / 264 at 2^28.
bool dense_pattern(uint32_t w, uint32_t L, uint32_t P, uint32_t pattern, uint64_t n)
{
    const uint64_t bytes = n * w;
    if (bytes <= (w == 8 ? 40ull << 20 : w == 2 ? 3ull << 19 : 3ull << 20)) return false;
    const bool late = w == 8 && bytes <= 96ull << 20;
    if (P * 100 < L * (late ? 70u : w == 1 || w == 8 ? 30u : 36u)) return false;
    uint32_t runs = 0; // of selected elements in a period
    for (uint32_t i = 0; i < L; ++i) runs += (pattern >> i & 1u) && !(pattern >> (i ? i - 1 : L - 1) & 1u);
    return !(w > 1 && P * w >= 32 * runs && P * 100 <= L * 55u);
}

// CTAs of the dense kernel per SM. 3 keep enough loads in flight for what is mostly read; where as
// much is written, 2 disturb the memory less: 4 bytes 0.375 217 (3) / 249 (2), 0.5 272 / 245, 0.97
// 364 / 322; 8 bytes 0.375 215 / 239, 0.5 273 / 250, 0.97 369 / 325. The 1- and 2-byte forms are
// held back by their instructions: 1 byte 0.97 88 / 100, 2 bytes 0.67 151 / 170, 0.97 188 / 172.
uint32_t dense_ctas_per_sm(uint32_t w, uint32_t L, uint32_t P)
{
    if (w == 1) return DENSE_CTAS;
    return P * 100 >= L * (w == 2 ? 85u : 45u) ? 2u : DENSE_CTAS;
}

template <typename T>
cudaError_t launch_t(const void* in, void* out, uint64_t n, uint32_t pattern, uint32_t L, uint32_t P, uint64_t count,
                     uint64_t* d_count, int sms, cudaStream_t s)
{
    constexpr uint64_t GROUP = 8 * PATTERN_RUNS * 32 * (sizeof(T) < 4 ? 4 / sizeof(T) : 1); // outputs per CTA and iteration
    uint64_t blocks = (count + GROUP - 1) / GROUP;
    const uint64_t cap = static_cast<uint64_t>(sms) * PATTERN_CTAS<T>;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    const bool vec = (reinterpret_cast<uintptr_t>(out) & 3u) == 0;
    const bool apart = sizeof(T) * L >= 64 * P;
    if (P == L && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0) {
        uint64_t ctas = (n * sizeof(T) + 256 * 4 * 16 - 1) / (256 * 4 * 16);
        const uint64_t most = static_cast<uint64_t>(sms) * COPY_CTAS;
        if (ctas > most) ctas = most;
        k_pattern_all<<<static_cast<unsigned>(ctas), 256, 0, s>>>(static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out),
                                                                 n * sizeof(T), count, d_count);
        note_launch();
        return cudaGetLastError();
    }
    if (dense_pattern(sizeof(T), L, P, pattern, n) && (reinterpret_cast<uintptr_t>(in) & 15u) == 0) {
        uint64_t rep = 0;
        for (uint32_t i = 0; i < 64; ++i) rep |= static_cast<uint64_t>((pattern >> (i % L)) & 1u) << i;
        const uint64_t items = (n * sizeof(T) + ITEM_BYTES - 1) / ITEM_BYTES;
        uint64_t ctas = (items + DENSE_WARPS - 1) / DENSE_WARPS;
        const uint64_t most = static_cast<uint64_t>(sms) * dense_ctas_per_sm(sizeof(T), L, P);
        if (ctas > most) ctas = most;
        // With an even number per period the lanes' elements fall into step on few banks, unless the
        // period divides a lane's elements (us, plain / swizzled stage: 2 bytes, 2 of 3 237 / 142, 2 of 5
        // 169 / 135, 3 of 7 131 / 139; 4 bytes, 2 of 5 249 / 226, 4 of 8 256 / 270)
        constexpr bool CAN = sizeof(T) == 2 || sizeof(T) == 4;
        const auto kernel = CAN && P % 2 == 0 && (L & (L - 1)) != 0 ? k_pattern_dense<T, CAN> : k_pattern_dense<T, false>;
        kernel<<<static_cast<unsigned>(ctas), DENSE_WARPS * 32, 0, s>>>(static_cast<const uint8_t*>(in),
                                                                        static_cast<uint8_t*>(out), n, pattern, rep, L, P,
                                                                        count, d_count);
        note_launch();
        return cudaGetLastError();
    }
    const T* ti = static_cast<const T*>(in);
    T* to = static_cast<T*>(out);
    const unsigned g = static_cast<unsigned>(blocks);
    if (vec && apart) k_pattern<T, true, true><<<g, 256, 0, s>>>(ti, to, pattern, L, P, count, d_count);
    else if (vec) k_pattern<T, true, false><<<g, 256, 0, s>>>(ti, to, pattern, L, P, count, d_count);
    else if (apart) k_pattern<T, false, true><<<g, 256, 0, s>>>(ti, to, pattern, L, P, count, d_count);
    else k_pattern<T, false, false><<<g, 256, 0, s>>>(ti, to, pattern, L, P, count, d_count);
    note_launch();
    return cudaGetLastError();
}

} // namespace

uint64_t pattern_count(uint64_t n, uint32_t pattern, uint32_t L)
{
    const uint32_t pm = L >= 32 ? pattern : (pattern & ((1u << L) - 1u));
    const uint32_t rem = static_cast<uint32_t>(n % L);
    const uint32_t partial = rem ? (pm & ((1u << rem) - 1u)) : 0u;
    return (n / L) * static_cast<uint64_t>(__builtin_popcount(pm)) + static_cast<uint64_t>(__builtin_popcount(partial));
}

} // namespace cs

using namespace cs;

extern "C" {

int compressstore_pattern(const void* d_in, void* d_out, uint64_t n, uint32_t elem_bytes, uint32_t pattern,
                          uint32_t pattern_length, uint64_t* d_count, cs_stream_t stream)
{
    if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return CS_ERR_INVALID_VALUE;
    if (pattern_length < 1 || pattern_length > 32 || !d_count) return CS_ERR_INVALID_VALUE;
    if (n > (1ull << 40) - 1) return CS_ERR_NOT_SUPPORTED;
    if (reinterpret_cast<uintptr_t>(d_count) & 7u) return CS_ERR_MISALIGNED;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t pm = pattern_length >= 32 ? pattern : (pattern & ((1u << pattern_length) - 1u));
    const uint64_t count = pattern_count(n, pm, pattern_length);
    if (count == 0) {
        const cudaError_t e = cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s);
        return e == cudaSuccess ? CS_SUCCESS : CS_ERR_CUDA;
    }
    if (!d_in || !d_out) return CS_ERR_INVALID_VALUE;
    if ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_out)) & (elem_bytes - 1u))
        return CS_ERR_MISALIGNED;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return CS_ERR_NO_DEVICE;
    const uint32_t P = static_cast<uint32_t>(__builtin_popcount(pm));
    cudaError_t e;
    switch (elem_bytes) {
        case 1: e = launch_t<uint8_t>(d_in, d_out, n, pm, pattern_length, P, count, d_count, sms, s); break;
        case 2: e = launch_t<uint16_t>(d_in, d_out, n, pm, pattern_length, P, count, d_count, sms, s); break;
        case 4: e = launch_t<uint32_t>(d_in, d_out, n, pm, pattern_length, P, count, d_count, sms, s); break;
        default: e = launch_t<uint64_t>(d_in, d_out, n, pm, pattern_length, P, count, d_count, sms, s); break;
    }
    return e == cudaSuccess ? CS_SUCCESS : (e == cudaErrorMemoryAllocation ? CS_ERR_OUT_OF_MEMORY : CS_ERR_CUDA);
}

} // extern "C"
