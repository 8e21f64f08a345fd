// cs_batch.cu — the batched form: a plan over many columns of uneven length and width.
//
// Each column takes the 3-pass hybrid or the 1-pass form, as the
// batch table of the autotuner says for its (width, size, selectivity) bucket; each pass is
// ONE launch for all the columns that take it: the reduce-then-scan popcount + prefix kernel
// walks a flat list of the 3-pass columns' 2^18-element blocks, one writeout per element width
// walks that width's 128 KB units and sparse 16K-element items over every SM, and one 1-pass
// kernel per width walks the 1-pass columns' units (decoupled look-back confined to each column). Work-to-column maps and column
// descriptors are built on the host once (cs_plan.cu) and uploaded with the plan, so a unit
// finds its column with one load. The launches can be captured in a CUDA graph.
//
// Selectivity is measured when the plan is built (CS_ALGO_AUTO, and only when the table has a
// 1-pass entry): one popcount pass over the masks into plan-owned count words. The choice
// changes speed, never results, so masks that change between runs stay correct.
#include <algorithm>
#include <vector>

#include <cuda_runtime.h>

#include "compressstore.h"
#include "cs_internal.cuh"
#include "cs_plan.h"
#include "cs_tuning.h"

using namespace cs;

struct cs_batch {
    int device = 0;
    int sms = 0;
    std::vector<uint64_t*> empty_counts; // d_count of n == 0 columns
    void* dmem = nullptr;
    size_t device_bytes = 0;
    PlanLayout layout;
    PlanDevice dev;
    PlanCounts counts;
    uint32_t grid1[4] = {0, 0, 0, 0};
    uint32_t idle8 = 0; // idle warps per CTA of the 8-byte columns' writeout
    uint32_t one_pass_cols = 0;
    std::vector<cs_column> cols; // for the per-call loop
    uint64_t timeout_ns = 2000000000ull;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint32_t kernels_per_run = 0;
};

namespace {

// Least payload the 3-pass columns of a mixed plan must hold to keep their form (about the
// bytes HBM moves in the 40 us their extra launches take).
constexpr uint64_t PLAN_3PASS_MIN_BYTES = 256ull << 20;
// ... and the payload from which on a plan takes one form (103 columns of 303 MB, both / 3-pass: 110 / 97 us).
constexpr uint64_t PLAN_LARGE_BYTES = 272ull << 20;

// Columns of one width are one launch in the 1-pass form and two in the 3-pass form, which shows where there is
// little to do, and in the middle, where the second launch waits for the first's tail. 1-pass / 3-pass, us, by
// plan: columns up to 2^14 elements, 4 bytes 1 column 10.3 / 11.6, 32 10.3 / 12.3, 256 15.2 / 17.5, 8 bytes 8.9 / 11.3,
// 10.3 / 12.3, 14.2 / 16.4, 2 bytes 1 10.9 / 12.3, 64 13.0 / 12.3, 256 16.4 / 18.4; 30 to 80 MB with 0.5 selected, 4 bytes
// 4 columns 20.6 / 22.6, 32 31.0 / 34.6, 256 24.9 / 26.5 (0.1: 18.7 / 19.9, 26.7 / 30.7, 22.7 / 24.4; 0.01: 18.5 / 14.3), 8 bytes 2
// 19.7 / 22.6, 16 32.2 / 33.7, 17 MB 4 15.1 / 16.4 (0.1: 18.3 / 17.8, 25.3 / 28.5), 2 bytes 32 24.7 / 26.6 (0.1: 22.7 / 22.6). 17 MB, 4 bytes
// 15.9 / 15.9 and 17.9 / 16.4, 100 MB 8 bytes 39.0 / 37.3; several widths: 4 and 8 bytes 34 MB 30.5 / 26.6. 1-byte
// columns are placed faster by the 3-pass form's warps at every size (14.3 / 12.3).
bool plan_one_launch(uint32_t widths, uint32_t columns, uint64_t longest, uint64_t bytes, double selected)
{
    if (widths != 2 && widths != 4 && widths != 8) return false; // (a sum of several is none of them)
    if (longest <= 1u << 14) return widths > 2 || columns <= 8 || columns > 128;
    return bytes >= (widths == 8 ? 16u << 20 : 28u << 20) && bytes <= 80u << 20 && selected >= (widths == 4 ? 0.05 : 0.3);
}

// Idle warps of the writeout (idle_warps in cs_writeout.cu) for the plan's 3-pass columns of 8 bytes, by what is
// selected of them when the plan is made: for 512 MB and more of them in columns of 11 MB and more on average. us with
// all warps / with idle ones, 0.85 to 0.95 selected: 16 columns 250 MB 87.5 / 89.9, 400 MB 139.7 / 134.1, 1.5 GB 502 / 457;
// 64 columns 550 MB 178.9 / 182.3, 750 MB 246.9 / 241.1, 1.5 GB 504 / 462; 128 columns 750 MB 239.8 / 244.8, 1.5 GB 496 /
// 467; 256 columns 400 MB 137 / 144, 1 GB 313 / 328. Plans of 4-byte columns lose (64 columns, 750 MB 252 / 259).
uint32_t idle_warps_of(const cs_column* cols, uint32_t ncols, const std::vector<uint8_t>& one_pass, const std::vector<double>& sel)
{
    double elems = 0.0, selected = 0.0, columns = 0.0;
    for (uint32_t i = 0; i < ncols; ++i) {
        if (one_pass[i] || cols[i].elem_bytes != 8 || !cols[i].n) continue;
        columns += 1.0;
        elems += static_cast<double>(cols[i].n);
        selected += sel[i] * static_cast<double>(cols[i].n);
    }
    const double bytes = elems * 8;
    return bytes >= 512.0 * (1 << 20) && bytes >= columns * 11.0 * (1 << 20) && selected >= 0.75 * elems ? 2u : 0u;
}

inline int to_status(cudaError_t e)
{
    if (e == cudaSuccess) return CS_SUCCESS;
    if (e == cudaErrorMemoryAllocation) return CS_ERR_OUT_OF_MEMORY;
    return CS_ERR_CUDA;
}

int run_direct(cs_batch* b, cudaStream_t s)
{
    for (uint64_t* c : b->empty_counts) {
        cudaError_t e = cudaMemsetAsync(c, 0, sizeof(uint64_t), s);
        if (e != cudaSuccess) return to_status(e);
    }
    return plan_launch(b->dev, b->counts, b->sms, b->timeout_ns, s, b->grid1, 0, b->idle8);
}

// Selected fraction of every column, from one reduce-then-scan popcount pass over the masks
// (into count words of a temporary plan, so nothing of the caller's is written). The temporary
// plan lies in *dmem, allocated here with the *room that the plan itself needs whatever the
// columns' forms turn out to be: device allocations are most of the time that making a plan takes
// (0.35 ms each, and 0.3 ms to free one, beside 0.2 ms of other work for 256 columns).
int measure_selectivity(const cs_column* cols, uint32_t ncols, int sms, cudaStream_t s, std::vector<double>& sel,
                        void** dmem, size_t* room)
{
    sel.assign(ncols, 0.0);
    std::vector<ColumnDesc> desc;
    std::vector<uint64_t> chunk_base;
    PlanCounts c;
    constexpr uint32_t ROW_LOG2 = 12; // whole 4096-element rows: only the counts are wanted
    int st = plan_columns(cols, ncols, desc, chunk_base, c, nullptr, nullptr, ROW_LOG2);
    if (st != CS_SUCCESS) return st;
    if (!c.tiles) return CS_SUCCESS;
    const PlanLayout L = plan_layout(c, true);
    PlanCounts c3, c1;
    const std::vector<uint8_t> all1(ncols, 1);
    std::vector<ColumnDesc> desc_unused;
    std::vector<uint64_t> base_unused;
    if ((st = plan_columns(cols, ncols, desc_unused, base_unused, c3, nullptr)) != CS_SUCCESS) return st;
    if ((st = plan_columns(cols, ncols, desc_unused, base_unused, c1, nullptr, &all1)) != CS_SUCCESS) return st;
    const size_t bytes = std::max(L.total, plan_layout(c3, false).total + plan_layout(c1, false).total);
    if (cudaMalloc(dmem, bytes) != cudaSuccess) {
        cudaGetLastError();
        *dmem = nullptr;
        return CS_ERR_OUT_OF_MEMORY;
    }
    *room = bytes;
    const PlanMaps m = plan_maps(c);
    const PlanDevice d = plan_device(static_cast<uint8_t*>(*dmem), L, m);
    for (uint32_t i = 0; i < ncols; ++i) desc[i].d_count = d.counts + i;
    std::vector<uint8_t> img(m.bytes);
    plan_write_image(img.data(), m, d, desc, chunk_base);
    std::vector<uint64_t> counts(ncols, 0);
    cudaError_t e = launch_ws_init(d.hdr, L.total, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.maps, img.data(), img.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        BlockScanParams bp{};
        bp.cols = d.cols;
        bp.blk_col = d.tile_col;
        bp.num_blocks = c.tiles;
        bp.blk_sum = d.blk_sum;
        bp.blk_base = d.blk_base;
        bp.hdr = d.hdr;
        bp.chunk_log2 = ROW_LOG2;
        bp.keep_begin = d.keep_begin;
        bp.keep_end = d.keep_end;
        e = launch_popc_blocks(bp, sms, s);
    }
    if (e == cudaSuccess && ncols) e = cudaMemcpyAsync(counts.data(), d.counts, 8 * ncols, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return to_status(e); // (the caller frees *dmem)
    for (uint32_t i = 0; i < ncols; ++i)
        if (cols[i].n) sel[i] = static_cast<double>(counts[i]) / static_cast<double>(cols[i].n);
    return CS_SUCCESS;
}

} // namespace

extern "C" {

int cs_batch_create(cs_batch** out, const cs_column* cols, uint32_t ncols, const cs_config* cfg, cs_stream_t stream)
{
    if (!out || (!cols && ncols)) return CS_ERR_INVALID_VALUE;
    *out = nullptr;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    auto b = new cs_batch();
    int major = 0;
    if (cudaGetDevice(&b->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, b->device) != cudaSuccess || major != 10) {
        delete b;
        return CS_ERR_NO_DEVICE;
    }
    if (cfg && cfg->timeout_ns) b->timeout_ns = cfg->timeout_ns;
    const int algo = cfg ? cfg->algo : CS_ALGO_AUTO;
    if (algo != CS_ALGO_AUTO && algo != CS_ALGO_1PASS && algo != CS_ALGO_3PASS) {
        delete b;
        return CS_ERR_INVALID_VALUE;
    }
    b->cols.assign(cols, cols + ncols);

    // per column: 1-pass or 3-pass (forced by cfg->algo, else the batch table's bucket)
    std::vector<uint8_t> one_pass(ncols, algo == CS_ALGO_1PASS ? 1 : 0);
    size_t room = 0; // of b->dmem, if it is already there
    if (algo == CS_ALGO_AUTO && tune_batch_any_1pass()) {
        std::vector<double> sel;
        const int st = measure_selectivity(cols, ncols, b->sms, s, sel, &b->dmem, &room);
        if (st != CS_SUCCESS) {
            cudaFree(b->dmem);
            delete b;
            return st;
        }
        for (uint32_t i = 0; i < ncols; ++i)
            one_pass[i] = cols[i].n && tune_batch_lookup(cols[i].n, cols[i].elem_bytes, sel[i]) == CS_ALGO_1PASS;
        // A plan of both forms runs both chains of launches, one after the other (about 30 us on B200), so it takes
        // one form where it can: the 3-pass form if the columns that the table names 1-pass hold less than a
        // quarter of the payload, otherwise the 1-pass form if the 3-pass columns hold less than
        // PLAN_3PASS_MIN_BYTES (3-pass / 1-pass, us: 28 columns of 9 MB 16 / 26, 101 of 40 MB 28 / 33, 256 of 2.2 GB
        // 577 / 615). Larger plans with a quarter or more named 1-pass keep both, as the table says (both /
        // 3-pass, us: 40 columns of 369 MB 117 / 112, 128 of 940 MB 265 / 255), and so do those between the two
        // lines (17 columns of 273 MB 90 / 82, 66 of 277 MB 115 / 101).
        uint64_t bytes3 = 0, bytes1 = 0, longest = 0;
        double selected = 0.0; // bytes
        uint32_t widths = 0, filled = 0;
        for (uint32_t i = 0; i < ncols; ++i) {
            const uint64_t bytes = cols[i].n * static_cast<uint64_t>(cols[i].elem_bytes);
            (one_pass[i] ? bytes1 : bytes3) += bytes;
            selected += sel[i] * static_cast<double>(bytes);
            if (!cols[i].n) continue;
            longest = std::max(longest, cols[i].n);
            widths |= cols[i].elem_bytes;
            ++filled;
        }
        const bool small = bytes3 < PLAN_3PASS_MIN_BYTES;
        if (bytes1 && (small || bytes1 + bytes3 >= PLAN_LARGE_BYTES)) {
            if (bytes1 < (bytes1 + bytes3) / 4) one_pass.assign(ncols, 0);
            else if (small)
                for (uint32_t i = 0; i < ncols; ++i) one_pass[i] = cols[i].n ? 1 : 0;
        }
        if (!bytes1 && plan_one_launch(widths, filled, longest, bytes3, bytes3 ? selected / static_cast<double>(bytes3) : 0.0))
            for (uint32_t i = 0; i < ncols; ++i) one_pass[i] = cols[i].n ? 1 : 0;
        b->idle8 = idle_warps_of(cols, ncols, one_pass, sel);
    }
    for (uint32_t i = 0; i < ncols; ++i) b->one_pass_cols += one_pass[i] && cols[i].n ? 1u : 0u;

    std::vector<ColumnDesc> desc;
    std::vector<uint64_t> chunk_base;
    int st = plan_columns(cols, ncols, desc, chunk_base, b->counts, &b->empty_counts, &one_pass);
    if (st != CS_SUCCESS) {
        cudaFree(b->dmem);
        delete b;
        return st;
    }
    b->layout = plan_layout(b->counts, false);
    cudaError_t e = cudaSuccess;
    if (b->layout.total > room) {
        cudaFree(b->dmem);
        b->dmem = nullptr;
        room = b->layout.total;
        e = cudaMalloc(&b->dmem, room);
    }
    b->device_bytes = room;
    if (e != cudaSuccess) {
        cudaGetLastError();
        delete b;
        return CS_ERR_OUT_OF_MEMORY;
    }
    const PlanMaps maps = plan_maps(b->counts);
    b->dev = plan_device(static_cast<uint8_t*>(b->dmem), b->layout, maps);
    std::vector<uint8_t> img(maps.bytes);
    plan_write_image(img.data(), maps, b->dev, desc, chunk_base);
    e = launch_ws_init(b->dev.hdr, b->layout.total, s); // zeroes everything, writes the header
    if (e == cudaSuccess && !img.empty())
        e = cudaMemcpyAsync(b->dev.maps, img.data(), img.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFree(b->dmem);
        delete b;
        return to_status(e);
    }
    // persistent grids (also applies the kernels' shared-memory attribute outside any capture)
    for (int wi = 0; wi < 4; ++wi) {
        b->grid1[wi] = plan_grid(1u << wi, b->counts.units1[wi], b->sms);
    }
    b->kernels_per_run = plan_kernels(b->counts);
    *out = b;
    return CS_SUCCESS;
}

int cs_batch_run(cs_batch* b, cs_stream_t stream)
{
    if (!b) return CS_ERR_INVALID_VALUE;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (b->exec) {
        cudaError_t e = cudaGraphLaunch(b->exec, s);
        if (e == cudaSuccess) note_launch(b->kernels_per_run);
        return to_status(e);
    }
    return run_direct(b, s);
}

int cs_batch_graph(cs_batch* b, cs_stream_t stream)
{
    if (!b) return CS_ERR_INVALID_VALUE;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (!s) return CS_ERR_INVALID_VALUE; // the legacy default stream cannot be captured
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return to_status(e);
    const uint64_t before = cs_launch_count();
    const int st = run_direct(b, s);
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(s, &g);
    note_launch(0 - (cs_launch_count() - before)); // captured, not executed
    if (st != CS_SUCCESS) {
        if (g) cudaGraphDestroy(g);
        return st;
    }
    if (e != cudaSuccess) return to_status(e);
    e = cudaGraphInstantiate(&b->exec, g, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return to_status(e);
    }
    b->graph = g;
    return CS_SUCCESS;
}

int cs_batch_check(cs_batch* b, cs_stream_t stream)
{
    if (!b) return CS_ERR_INVALID_VALUE;
    return cs_workspace_check(b->dev.hdr, stream);
}

int cs_batch_run_per_call(cs_batch* b, cs_stream_t stream)
{
    if (!b) return CS_ERR_INVALID_VALUE;
    for (const cs_column& c : b->cols) {
        const int st = compressstore(c.d_in, c.d_mask, c.d_out, c.n, c.elem_bytes, c.d_count, stream);
        if (st != CS_SUCCESS) return st;
    }
    return CS_SUCCESS;
}

uint32_t cs_batch_one_pass_columns(const cs_batch* b)
{
    return b ? b->one_pass_cols : 0u;
}

uint64_t cs_batch_device_bytes(const cs_batch* b)
{
    return b ? b->device_bytes : 0;
}

uint32_t cs_batch_launches(const cs_batch* b)
{
    return b ? (b->exec ? 1u : b->kernels_per_run) : 0u;
}

int cs_batch_destroy(cs_batch* b)
{
    if (!b) return CS_SUCCESS;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->dmem) cudaFree(b->dmem);
    delete b;
    return CS_SUCCESS;
}

} // extern "C"
