// B200 (sm_100a) permutohedral-lattice filter: kernels and the C ABI of include/pl_lattice.h.
//
// Pipeline of one call (whole batch in every launch, nothing synchronises with the host):
//
//   clear_header    zeroes the counters; in calls without a sketch, and with direct indexing, clears the table too.
//   build_tiles     one CTA per tile of TP points: features -> enclosing simplex -> pd+1 vertex keys
//                   per point; the tile's keys are de-duplicated in a shared-memory hash; the
//                   distinct keys become a contiguous run of "entries" in a global list and every
//                   splat records the 16-bit index of its entry inside the tile.
//   clear_table     calls with a sketch: sizes the global hash table (on the device) from the entry count or from
//                   build_tiles' sketch of the vertices, and clears it and the filter in front of it.
//   insert_entries  one CAS per entry into the table; the first entry of a key owns a new vertex, whose
//                   neighbour slots the same launch initialises.  Up to pd 5 insert_keys, into slots that hold the key.
//   link_neighbours entry -> vertex index; value rows zeroed; then the +-1 neighbours of every vertex along each
//                   of the pd+1 axes: one table lookup per vertex and axis fills both directions.
//   splat_tiles     one CTA per tile: input block staged in shared memory (bulk async copies), splats
//                   sorted by entry, runs summed in registers, vector reductions into the vertex rows.  Tiles with
//                   few entries, up to pd 4: columns of points instead of the sort.
//   blur_axis       pd+1 launches: V'[v] = (V[n1] + 2 V[v] + V[n2]) / 4, Jacobi, ping-pong buffers.  Medium-sized
//                   lattices: two passes a launch (blur_pair).
//   slice_tiles     one CTA per tile: the tile's vertex rows staged in shared memory, each point
//                   interpolates, divides by the homogeneous channel and writes its output row.  Rows of one
//                   float4 (slice_points): straight from global memory.
//
// Small lattices take one launch for the three index kernels and one for all blur passes (small.cuh); spatial-only calls
// index their vertices without hashing (direct_index.cuh).
//
// A table slot is one 64-bit word (beyond pd 5; else see KeySlot): 32-bit hash tag | index of the entry that created the vertex, which becomes the
// vertex's own index when the creator's round ends.  Full keys are compared through the entry list, which a previous
// launch has completely written, or through the vertex's key, so there are no locks, no waiting and no duplicate
// vertices.  All device loops are bounded.
//
// Device code lives in the headers included below (one translation unit); this file holds the host
// side: geometry and workspace layout, launches, and the extern "C" entry points.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <mutex>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <thread>
#include <utility>
#include <vector>

#include "common.cuh"
#include "lattice_build.cuh"
#include "direct_index.cuh"
#include "splat.cuh"
#include "blur_slice.cuh"
#include "small.cuh"
#include "export.cuh"
#include "fp64.cuh"
#include "crf.cuh"
#include "smem_limit.h"

namespace pl {

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
static thread_local char g_cuda_error[256] = "";
// Stage-boundary events for the next filter call of this thread (pl_profile_next_call); consumed by it.
static thread_local cudaEvent_t* g_stage_events = nullptr;

// Kernel launches issued by the library since it was loaded (pl_launch_count): memsets and event
// records are not counted.
static std::atomic<unsigned long long> g_launches{0};
#define PL_COUNT_LAUNCHES(n) g_launches.fetch_add((n), std::memory_order_relaxed)

static int cuda_fail(cudaError_t e, const char* where) {
    snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s", where, cudaGetErrorString(e));
    return PL_CUDA_ERROR;
}

#define PL_CUDA(call)                                   \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

// Pinned words in which watched calls (pl_watch_next_call) report their counters: a 64-byte line each, handed
// to a thread when it first watches a call and taken back when the thread ends (the pool is as large as the
// number of threads that ever watched at the same time, in pages of 64 lines).  The sequence number, which goes
// with the line, tells its reports apart: a late one of a call that was given up on is not mistaken for the
// next call's.
struct alignas(64) WatchLine {
    u64 words[2];   // what the device writes (see Watch): the report, and the status bits of a failure after it
    u32 seq;
};
static std::mutex g_watch_mutex;
static std::vector<WatchLine*>& watch_pages() {   // every page of 64 lines there is
    static std::vector<WatchLine*>* pages = new std::vector<WatchLine*>();
    return *pages;
}
static std::vector<WatchLine*>& watch_pool() {
    static std::vector<WatchLine*>* pool = new std::vector<WatchLine*>();   // outlives every thread
    return *pool;
}
struct Watcher {
    WatchLine* line = nullptr;
    bool armed = false;     // the next call of this thread reports
    bool launched = false;  // a call that reports has been queued
    ~Watcher() {
        if (!line) return;
        std::lock_guard<std::mutex> lock(g_watch_mutex);
        watch_pool().push_back(line);
    }
};
static thread_local Watcher g_watcher;

static int take_watch_line(WatchLine** out) {
    std::lock_guard<std::mutex> lock(g_watch_mutex);
    std::vector<WatchLine*>& pool = watch_pool();
    if (pool.empty()) {
        void* p = nullptr;
        PL_CUDA(cudaHostAlloc(&p, 64 * sizeof(WatchLine), cudaHostAllocPortable | cudaHostAllocMapped));
        memset(p, 0, 64 * sizeof(WatchLine));
        watch_pages().push_back(static_cast<WatchLine*>(p));
        for (int i = 0; i < 64; i++) pool.push_back(static_cast<WatchLine*>(p) + i);
    }
    *out = pool.back();
    pool.pop_back();
    return PL_OK;
}

// What a call passes to its link kernel: where to report, or nothing.  A call that is being captured never reports: the
// graph would write into the line at every replay.
static Watch take_watch(cudaStream_t st) {
    Watch w = {nullptr, 0u};
    if (!g_watcher.armed) return w;
    g_watcher.armed = false;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) {
        w.words = g_watcher.line->words;
        w.seq = g_watcher.line->seq;
        g_watcher.launched = true;
    }
    return w;
}
static int code_of(u64 status_bits) {
    int code = PL_OK;
    for (int c = PL_INVALID_ARGUMENT; c <= PL_INTERNAL_ERROR; c++)
        if (status_bits & (1u << c)) code = c;
    return code;
}
// The failure after its report, if any, of a call that reported to this line; told once.
static int take_late_failure(WatchLine* line) {
    return code_of(__atomic_exchange_n(&line->words[1], 0ull, __ATOMIC_ACQ_REL));
}
// In every filter and build entry point: the watch is for this call, however far it gets, and never for a later one.
struct WatchScope {
    ~WatchScope() { g_watcher.armed = false; }
};

// Kernel launch with the error check of every other runtime call.  overlap: with programmatic stream
// serialisation, i.e. the kernel may become resident while the kernel before it in the stream drains (it waits
// in after_previous_kernel() until that kernel has finished).
template <typename... Params, typename... Args>
static cudaError_t launch_kernel(bool overlap, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    if (overlap) {
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
#define PL_LAUNCH(kernel, grid, block, smem, st, ...) \
    PL_CUDA(launch_kernel(false, kernel, dim3(grid), dim3(block), smem, st, __VA_ARGS__))
// A launch that may overlap the tail of the kernel before it: all but clear_header, which starts a call, and those whose callers say why not (an
// apply
// and a CRF step start with a kernel that overlaps whatever came before the call).
// What each gave when it was measured by itself, all others as they are now, us a call or step, plain / overlapped: the blur passes after one
// another, 16 and 2 items of 512x512 x 21, 2023 / 2007 and 353 / 342; the slice after the last pass and the splat after the link 2002 and 335;
// clear_table after the build 1993 and 331; the insert after clear_table 1992 and 328.  The link after the insert and the first
// blur pass after the splat, which gain only where the insert and the splat release them at their end (see
// wait_for_previous_kernel): 800x1200 x 3 176.6 / 172.3, 1024x1024 grey by RGB, forward + backward, 306.9 / 299.4, five CRF steps on
// 375x500 x 21 427 / 411 (and 408 with the index stage of the two kept lattices), two volumes of 111x128x120 509 / 502, 8 x 512x512 x 21 without a
// guide 424 / 415, 16 x 512x512 x 21 1764 / 1764.
#define PL_LAUNCH_AFTER(overlap, kernel, grid, block, smem, st, ...) \
    PL_CUDA(launch_kernel((overlap), kernel, dim3(grid), dim3(block), smem, st, __VA_ARGS__))

// The header and the sketch behind it.
constexpr size_t HEADER_BYTES = sizeof(Header) + sizeof(u32) * SKETCH_WORDS;

// Sampling of the sketch (see SKETCH_LOG2): so that a lattice of max_entries vertices sets about half its bits.  A call keeps one when its table is
// cleared by a launch of its own, which sizes it by the sketch (see ClearTable: bounds of more than 2^19 entries).
static int sketch_shift_of(u64 max_entries) {
    int shift = 0;
    while (shift < 20 && (max_entries >> shift) > (1ull << (SKETCH_LOG2 - 1))) shift++;
    return shift;
}

static size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

static int tp_of(int pd) { return pd <= 8 ? 256 : 128; }
static int kw_of(int pd) { return (pd + 1 + 3) / 4; }
// 8-byte words of a tile's sorted splat list (Cfg<PD>::SREC)
static int srec_words_of(int pd) {
    const int splats = tp_of(pd) * (pd + 1), wl = 8 * (pd + 1);
    return splats + 2 * (splats / wl);
}

static bool pd_supported(int pd) {
    return pd == 1 || pd == 2 || pd == 3 || pd == 4 || pd == 5 || pd == 6 || pd == 7 || pd == 8 ||
           pd == 16;
}

// src/PermutohedralLatticeCPU.h:194-217, T = float: double arithmetic rounded to float.
static void scale_factors(int pd, float* out) {
    float inv_std_dev = (float)((pd + 1) * sqrt(2.0 / 3));
    for (int i = 0; i < pd; i++)
        out[i] = (float)(1.0 / sqrt((double)((i + 1) * (i + 2))) * (double)inv_std_dev);
}

// T = double: standard deviations and scale factors (src/PermutohedralLatticeCPU.h:194-217) in double.
static void set_geom_f64(Geom& g, int pd, double spatial_std, double feature_std) {
    g.spatial_std_d = spatial_std;
    g.feature_std_d = feature_std;
    const double inv_std_dev = (pd + 1) * sqrt(2.0 / 3);
    for (int i = 0; i < pd; i++) g.scale_d[i] = 1.0 / sqrt((double)((i + 1) * (i + 2))) * inv_std_dev;
}

static int make_geom(Geom& g, int batch, int n, int pd, int n_sdims, const int* sdims, int R,
                     float spatial_std, float feature_std, bool from_positions) {
    memset(&g, 0, sizeof(g));
    g.batch = batch;
    g.n = n;
    g.from_positions = from_positions ? 1 : 0;
    g.lattice_items = 1;
    g.row_step = 1;
    g.n_sdims = n_sdims;
    g.R = R;
    g.spatial_std = spatial_std;
    g.feature_std = feature_std;
    // Division through a correctly rounded reciprocal and one fused correction gives the IEEE quotient
    // as long as nothing leaves the normal range; keep the plain divide for extreme sigmas.
    auto tame = [](float v) { return std::isfinite(v) && std::fabs(v) >= 1e-18f && std::fabs(v) <= 1e18f; };
    g.spatial_rcp = 1.0f / spatial_std;
    g.feature_rcp = 1.0f / feature_std;
    g.rcp_div = (tame(spatial_std) && tame(feature_std)) ? 1 : 0;
    const int tp = tp_of(pd);
    if (from_positions || n_sdims < 2) {
        g.W = n; g.H = 1; g.outer = 1;
        g.TX = tp; g.TY = 1;
    } else {
        g.W = sdims[n_sdims - 1];
        g.H = sdims[n_sdims - 2];
        g.outer = 1;
        for (int i = 0; i < n_sdims - 2; i++) g.outer *= sdims[i];
        g.TX = 16;
        while (g.TX > 1 && g.TX / 2 >= g.W) g.TX /= 2;   // narrow images: narrower, taller tiles
        g.TY = tp / g.TX;
    }
    for (int i = 0; i < n_sdims; i++) g.sdims[i] = sdims[i];
    g.tiles_x = (g.W + g.TX - 1) / g.TX;
    g.tiles_y = (g.H + g.TY - 1) / g.TY;
    long long per_item = (long long)g.tiles_x * g.tiles_y * g.outer;
    long long total = per_item * batch;
    if (total > 0x7FFFFFFFll) return PL_INVALID_ARGUMENT;
    g.tiles_per_item = (int)per_item;
    g.num_tiles = (int)total;
    g.tx_log2 = 0;
    while ((1 << g.tx_log2) < g.TX) g.tx_log2++;
    // Under a guide that is flat, a tile of 16 x 16 points has about (pd + 1) (1 + 0.7 * 16 / spatial_std)^2 entries (0.6 to
    // 0.8 for 0.7 with pd 2 to 4, spatial_std 1.5 to 25, from the oracle's lattices): half as many again.
    const double std_abs = std::fabs((double)spatial_std), across = 1.0 + (std_abs > 1e-3 ? 11.2 / std_abs : 1e4);
    g.calm_entries = (int)std::min(1.5 * (pd + 1) * across * across, 65536.0);
    g.grid3 = (g.tiles_y <= 65535 && (long long)batch * g.outer <= 65535) ? 1 : 0;
    scale_factors(pd, g.scale);
    return PL_OK;
}

// real_bytes: 4 for float calls, 8 for double calls (wider weights and value rows, no fixed-point sums).
// with_fixed_point: the workspace also holds the 64-bit sums of the deterministic mode (float calls only).
// with_sorted: it also holds every tile's splats sorted (float calls only; used by lattices built to be applied later).
static int make_layout(Layout& L, const Geom& g, int pd, int vd, int64_t max_entries_arg, int real_bytes = 4,
                       bool with_fixed_point = false, bool with_sorted = true) {
    const u64 S = (u64)g.batch * (u64)g.n * (u64)(pd + 1);
    if (S >= 0x7FFFFFF0ull) return PL_INVALID_ARGUMENT;
    u64 E = (max_entries_arg <= 0 || (u64)max_entries_arg > S) ? S : (u64)max_entries_arg;
    if (E < 1) E = 1;
    L.max_entries = E;
    u64 slots = 1024;
    while (slots < 2 * E) slots <<= 1;
    L.table_slots = slots;
    L.key_slots = pd <= 5;
    L.index_words = 2 * slots;
    const size_t tile_splats = (size_t)tp_of(pd) * (pd + 1);
    size_t off = align_up(HEADER_BYTES);
    L.tile_info = off; off += align_up(sizeof(int2) * (size_t)g.num_tiles);
    L.rec = off;       off += align_up(sizeof(u16) * tile_splats * (size_t)g.num_tiles);
    L.rec_w = off;     off += align_up((size_t)real_bytes * tile_splats * (size_t)g.num_tiles);
    L.srec = off;      // the splats of every tile sorted by entry (float calls: what their splat kernels walk)
    if (real_bytes == 4 && with_sorted) off += align_up(sizeof(uint2) * (size_t)srec_words_of(pd) * (size_t)g.num_tiles);
    L.list_keys = off; off += align_up(sizeof(u64) * kw_of(pd) * E);
    L.list_ref = off;  off += align_up(sizeof(u32) * E);
    L.vid = off;       off += align_up(sizeof(u32) * E);
    L.vkeys = off;     off += align_up(sizeof(u64) * kw_of(pd) * E);
    L.table = off;     off += L.key_slots ? 0 : align_up(sizeof(u64) * slots);
    L.nbr = off;       off += align_up(sizeof(int) * 2 * (size_t)(pd + 1) * E);
    const size_t row_bytes = real_bytes == 8 ? sizeof(double) * (size_t)padded_vd_f64(vd)
                                             : sizeof(float) * (size_t)padded_vd(vd);
    L.v0 = off;        off += align_up(row_bytes * E);
    L.v1 = off;
    if (L.key_slots) {
        // The table lies where the second buffer of value rows does: nothing reads the table once the neighbours are
        // linked, nothing touches those rows before the first blur pass.  Rows of one float4 are shorter than the slots
        // of 16 bytes.  The scratch without allocation has a fixed size and takes what it always took: with slots of 8
        // bytes where it would be too small, never with fewer than two an entry (a lookup that finds nothing walks 2.5
        // slots of a table half full, 35 at a load of 0.88 and thousands close to 1).
        L.table = L.v1;
        if (!with_sorted && off + align_up(2 * sizeof(u64) * slots) > PL_STATIC_SCRATCH_BYTES) L.key_slots = false;
        off += align_up(std::max(row_bytes * (size_t)E, (size_t)((L.key_slots ? 2 : 1) * sizeof(u64) * slots)));
    } else {
        off += align_up(row_bytes * E);
    }
    L.v64 = off;       // deterministic mode sums (float calls only)
    if (real_bytes == 4 && with_fixed_point) off += align_up(sizeof(long long) * (size_t)padded_vd(vd) * E);
    L.total = off;
    return PL_OK;
}

// Developer switch (pl_debug_direct_index): 0 sends spatial-only calls through the hash table too.
static int g_direct_index_enabled = 1;

// The dense index of a spatial-only call (direct_bounds.h), if the call qualifies and the index fits the
// table region of the workspace (32-bit slots in the memory of the 64-bit hash slots).
static bool make_direct(Direct& d, const Geom& g, int pd, const Layout& L) {
    memset(&d, 0, sizeof(d));
    if (!g_direct_index_enabled || g.from_positions || g.R != 0 || pd != g.n_sdims) return false;
    return direct_bounds(d, pd, g.sdims, g.spatial_std, g.scale, g.batch, L.index_words);
}

// Where one lattice serves several items: whether a vertex's rows lie together, or an item's.  With an item's, conversion and blur have a row of
// blocks for every item, which have next to nothing to do in a small lattice, and ask for a vertex's neighbours once an item; with a
// vertex's, rows of one float4 share their lines with other items' and not with those of the tile's other vertices, and of large lattices
// more lines come from DRAM.  So by the bounds, of an item's entries and, for longer rows, of all rows.  us a call without a guide, an item's
// / a vertex's together: 65535x4x4 x 3 15180 / 181, 1024x8x8 x 3 136 / 24.5, 64x64x64 x 3 39 / 27, 300x5000 x 1 81 / 46 (these with the zeroing
// item by item too); bounds of 67 to 196 k entries an item, 8x512x512 x 1, theta 8, 65 / 58, theta 2 79 / 83, 1 128 / 139, 0.7 217 / 261, 16x300x300
// x 3, theta 2, 65 / 67; 8x512x512 x 10, theta 2 164 / 162, 1 372 / 362, 0.7 667 / 745, x 21, theta 3, 173 / 168, 1 585 / 585, 0.7 1291 / 1415,
// 2x1000x1000 x 21, theta 1, 606 / 620, 64x100x120 x 21, theta 1, 247 / 198, 3x100x100x100 x 10, theta 1, 940 / 803.
constexpr u64 TOGETHER_ENTRIES = 16384;
constexpr u64 TOGETHER_BYTES = 256u << 20;
static bool rows_together(const Layout& whole, const Layout& share, int vd) {
    const u64 row_bytes = sizeof(float) * (u64)padded_vd(vd);
    return share.max_entries <= TOGETHER_ENTRIES || (row_bytes > 16 && whole.max_entries * row_bytes <= TOGETHER_BYTES);
}

// The features of a spatial-only call are those of its grid, the same in every item: one lattice does for all, with its share of the
// bound, and value rows for every item.  The lattice's own geometry and layout, of one item; false: the call builds a lattice of all
// its items.  A share fits where the whole would have: entries are the same in every item.  us a call, forward + backward, an own
// lattice each / one: 8 x 512x512 x 21 414 / 334, 16 x 512x512 x 1 399 / 217; forward, 1024x8x8 x 3 28.5 / 24.5, 65535x4x4 x 3 424 / 181.
static bool one_for_all(const Geom& g, const Layout& L, int pd, int vd, Geom& one, Layout& share) {
    one = g;
    share = L;
    if (g.from_positions || g.R != 0 || pd != g.n_sdims || g.batch < 2 || L.max_entries < (u64)g.batch) return false;
    share.max_entries = L.max_entries / (u64)g.batch;
    while (share.table_slots > 1024 && share.table_slots / 2 >= 2 * share.max_entries) share.table_slots /= 2;
    one.lattice_items = g.batch;
    one.item_entries = (u32)share.max_entries;
    one.bound = (u32)L.max_entries;
    one.row_step = rows_together(L, share, vd) ? (u32)g.batch : 1u;
    one.batch = 1;
    one.num_tiles = one.tiles_per_item;
    one.grid3 = (one.tiles_y <= 65535 && one.outer <= 65535) ? 1 : 0;
    return true;
}

// What clear_header clears for the index stage (see ClearTable): the direct index, or all of the hash table.  A small lattice's table lies
// elsewhere.
static ClearTable table_to_clear(const Direct* direct, const Layout& L, void* table, bool small, bool beside_build) {
    ClearTable c = {nullptr, 0u};
    const u64 bytes = direct ? sizeof(u32) * direct->slots : (L.key_slots ? 16ull : 8ull) * L.table_slots;
    if (small || bytes > 16ull * (beside_build ? CLEAR_QUADS : CLEAR_QUADS_ALONE)) return c;
    c.table = static_cast<uint4*>(table);
    c.quads = (u32)((bytes + 15) / 16);   // (regions are 256-byte aligned: so is the end)
    return c;
}

// Launch grid of the tile kernels (see this_tile).
static dim3 tile_grid(const Geom& g) {
    if (g.grid3) return dim3((unsigned)g.tiles_x, (unsigned)g.tiles_y, (unsigned)(g.batch * g.outer));
    return dim3((unsigned)g.num_tiles, 1, 1);
}

static int g_num_sms = 0;
static int num_sms() {
    if (g_num_sms == 0) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
            sms = 148;
        g_num_sms = sms;
    }
    return g_num_sms;
}

// Raises a kernel's dynamic shared-memory limit (and sets its carve-out preference) when this call needs more than any
// call before it on the current device.
template <auto Kernel>
static int ensure_dynamic_smem(size_t bytes, bool max_carveout = false) {
    static SmemLimit limit;
    int dev = -1;
    PL_CUDA(cudaGetDevice(&dev));
    return limit.raise(dev, bytes, [&](size_t n) -> int {
        PL_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n));
        if (max_carveout)
            PL_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared));
        return PL_OK;
    });
}
#define PL_TRY(call)                     \
    do {                                 \
        const int rc_ = (call);          \
        if (rc_ != PL_OK) return rc_;    \
    } while (0)

// Rows of the per-tile shared-memory vertex-row cache of slice_tiles (48 KB of rows at most).
static int rows_cap_for(int pd, int vd) {
    const int splats = tp_of(pd) * (pd + 1);
    int cap = (48 * 1024) / (padded_vd(vd) * (int)sizeof(float));
    if (cap > splats) cap = splats;
    if (cap < 1) cap = 1;
    return cap;
}

// Widest row the splat stage takes: its tile's rows and twice its sorted list within 200 KB.  (The kernel's own need,
// SplatRows::bytes, is a little less.)
static int widest_vd(int pd) {
    const int tp = tp_of(pd);
    return ((200 * 1024 - 16 * tp * (pd + 1) - 4 * tp) / (4 * tp)) & ~3;
}

// The same of the deterministic splat: unpadded input rows and one and a half sorted lists within 200 KB.  (With its rows
// padded the kernel asks for up to 209,408 bytes, at pd 4 and 8, of the 227 KB that a block may have.)
static int widest_vd_fixed(int pd) {
    const int tp = tp_of(pd);
    return (200 * 1024 - 12 * tp * (pd + 1) - 4 * tp) / (4 * tp) + 1;
}

// True when every contiguous run of a tile's points starts on a 16-byte boundary and has a size that is
// a multiple of 16 bytes in a [points][channels] float array at `ptr`: then the tile's block can move
// by bulk asynchronous copies.
static bool bulk_rows_ok(const Geom& g, const void* ptr, int channels) {
    const long long row_bytes = 4ll * channels;
    return ((uintptr_t)ptr % 16 == 0) && (row_bytes * g.W) % 16 == 0 && (row_bytes * g.TX) % 16 == 0 &&
           (row_bytes * g.n) % 16 == 0 && (row_bytes * g.TX * g.TY) < (1ll << 31);
}

// link_neighbours: a row of blocks for each lattice axis, long enough that the rows run one after the other on a
// large lattice: threads then work on one axis of a stretch of vertices at a time, whose neighbours along that axis
// lie close together too.  (All axes at once, in rows that fill the GPU together, measured 96 instead of 72 us on
// the 16-image dense-CRF batch.)  On a small one, no more blocks than there can be vertices for.
template <int PD>
static dim3 link_grid(int wide, u64 max_entries) {
    const u64 blocks = (max_entries + 511) / 512;
    return dim3((unsigned)(blocks < (u64)wide ? blocks : (u64)wide), PD + 1, 1);
}

// Bulk copies into padded rows (splat_tiles_rows) also need 16-byte aligned landing zones inside the tile rows.
static bool bulk_staging_ok(const Geom& g, const float* input, int vd) {
    return bulk_rows_ok(g, input, vd - 1) && g.TX <= 16 && (g.TX * (padded_vd(vd) - (vd - 1))) % 4 == 0;
}

// splat for value dimension VD, fixed at compile time, or (VD = 0) any other.
// Rows of one float4 (VD <= 4) are summed by a thread each, wider ones by a group of lanes (splat.cuh).
template <int PD, int VD, bool PRE>
static int launch_splat_as(const Geom& g, const float* input, Header* hdr, const int2* tile_info, const u16* rec,
                           const float* rec_w, const uint2* srec, const u32* list_ref, float* v0, int vd,
                           cudaStream_t st) {
    if constexpr (VD > 0 && VD <= 4) {
        const size_t smem = SplatFast<PD, VD, PRE>::BYTES;
        PL_TRY((ensure_dynamic_smem<splat_tiles_fast<PD, VD, PRE>>(smem)));
        PL_LAUNCH_AFTER(true, (splat_tiles_fast<PD, VD, PRE>), tile_grid(g), Cfg<PD>::TP, smem, st, g, input, hdr, tile_info, rec, rec_w,
                                                                              srec, list_ref, v0, bulk_rows_ok(g, input, VD - 1) ? 1 : 0);
    } else {
        const size_t smem = SplatRows<PD, VD, PRE>::bytes(vd);
        if (vd > widest_vd(PD)) return PL_UNSUPPORTED_DIMS;
        // five CTAs per SM need nearly all of the SM's shared memory: ask for the largest carve-out
        PL_TRY((ensure_dynamic_smem<splat_tiles_rows<PD, VD, PRE, FloatSum, float>>(smem, true)));
        const bool bulk = bulk_staging_ok(g, input, vd);
        PL_LAUNCH_AFTER(true, (splat_tiles_rows<PD, VD, PRE, FloatSum, float>), tile_grid(g), Cfg<PD>::TP, smem, st, g, input, hdr,
                tile_info, rec, rec_w,
                                                                              srec, list_ref, v0, vd, bulk ? 1 : 0);
    }
    return PL_OK;
}

// The deterministic splat: fixed-point sums, rows of any width.
template <int PD, bool PRE>
static int launch_splat_fixed(const Geom& g, const float* input, Header* hdr, const int2* tile_info, const u16* rec,
                              const float* rec_w, const uint2* srec, const u32* list_ref, long long* v64, int vd,
                              cudaStream_t st) {
    const size_t smem = SplatRows<PD, 0, PRE>::bytes(vd);
    PL_TRY((ensure_dynamic_smem<splat_tiles_rows<PD, 0, PRE, FixedSum, long long>>(smem, true)));
    const bool bulk = bulk_staging_ok(g, input, vd);
    PL_LAUNCH_AFTER(true, (splat_tiles_rows<PD, 0, PRE, FixedSum, long long>), tile_grid(g), Cfg<PD>::TP, smem, st, g, input, hdr,
            tile_info, rec, rec_w,
                                                                          srec, list_ref, v64, vd, bulk ? 1 : 0);
    return PL_OK;
}

// presorted: the lattice was built for reuse (build_tiles with SORTED) and holds its splats sorted in srec
template <int PD, int VD>
static int launch_splat(const Geom& g, const float* input, Header* hdr, const int2* tile_info, const u16* rec,
                        const float* rec_w, const uint2* srec, bool presorted, const u32* list_ref, float* v0, int vd,
                        cudaStream_t st) {
    return presorted ? launch_splat_as<PD, VD, true>(g, input, hdr, tile_info, rec, rec_w, srec, list_ref, v0, vd, st)
                     : launch_splat_as<PD, VD, false>(g, input, hdr, tile_info, rec, rec_w, srec, list_ref, v0, vd, st);
}

// Whether the slice of wide rows overlaps the last blur pass.  With fewer tiles than SMs not: of a grid that starts
// while the pass leaves the GPU, four or five CTAs go to the first SMs that become free, and the others stay idle (12 k vertices of 2000
// points at pd 5, 21 channels: the slice 25 / 8 us, the call 88 / 74; 8 x 79x38 x 30 in double 33 / 15 and 81 / 66).  The small blur leaves most SMs free for it.  Narrow rows read
// too little for it to matter: the plain launch costs them 1 to 2 us.
static bool slice_overlap(const Geom& g, bool after_small_blur) {
    return after_small_blur || g.num_tiles >= num_sms();
}

// slice for rows of VP floats (CT > 0: of CT channels), or (VP = 0) of more than 32.
template <int PD, int VP, int CT = 0>
static int launch_slice(const Geom& g, float* output, const Header* hdr, const int2* tile_info, const u16* rec,
                        const float* rec_w, const u32* list_ref, const float* vsrc, int vd, Watch watch, bool overlap, cudaStream_t st) {
    if constexpr (VP == 4) {
        PL_LAUNCH_AFTER(true, (slice_points<PD, CT>), tile_grid(g), Cfg<PD>::TP, 0, st, g, output, hdr, tile_info, rec, rec_w, list_ref, vsrc, watch);
    } else if constexpr (VP > 0) {
        int rows_cap = SliceFast<PD, VP, CT>::ROWS_BYTES / (SliceFast<PD, VP>::RS * 4);
        if (rows_cap > Cfg<PD>::SPLATS) rows_cap = Cfg<PD>::SPLATS;
        const size_t smem = SliceFast<PD, VP>::bytes(rows_cap);
        PL_TRY((ensure_dynamic_smem<slice_tiles_fast<PD, VP, CT>>(smem)));
        PL_LAUNCH_AFTER(overlap, (slice_tiles_fast<PD, VP, CT>), tile_grid(g), Cfg<PD>::TP, smem, st, g, output, hdr, tile_info, rec, rec_w, list_ref, vsrc, vd - 1, rows_cap, bulk_rows_ok(g, output, vd - 1) ? 1 : 0, watch);
    } else {
        const int rows_cap = rows_cap_for(PD, vd);
        const size_t fixed = sizeof(float) * Cfg<PD>::TP * SliceCfg<PD>::PW + sizeof(int) * Cfg<PD>::TP;
        const size_t smem = sizeof(float) * (size_t)rows_cap * padded_vd(vd) + fixed;
        if (smem > 200 * 1024) return PL_UNSUPPORTED_DIMS;
        PL_TRY((ensure_dynamic_smem<slice_tiles_generic<PD>>(smem)));
        PL_LAUNCH_AFTER(overlap, (slice_tiles_generic<PD>), tile_grid(g), Cfg<PD>::TP, smem, st, g, output, hdr, tile_info, rec, rec_w,
                                                                        list_ref, vsrc, vd, rows_cap, watch);
    }
    return PL_OK;
}

// The instantiation of splat (slice) for value dimension vd.
#define PL_SPLAT_FOR(PD_, vd, ...)                  \
    ((vd) == 22  ? launch_splat<PD_, 22>(__VA_ARGS__) \
     : (vd) == 4 ? launch_splat<PD_, 4>(__VA_ARGS__)  \
     : (vd) == 3 ? launch_splat<PD_, 3>(__VA_ARGS__)  \
     : (vd) == 2 ? launch_splat<PD_, 2>(__VA_ARGS__)  \
                 : launch_splat<PD_, 0>(__VA_ARGS__))
#define PL_SLICE_FOR(PD_, vd, ...)                              \
    ((vd) == 22            ? launch_slice<PD_, 24, 21>(__VA_ARGS__) \
     : (vd) == 4           ? launch_slice<PD_, 4, 3>(__VA_ARGS__)   \
     : (vd) == 3           ? launch_slice<PD_, 4, 2>(__VA_ARGS__)   \
     : (vd) == 2           ? launch_slice<PD_, 4, 1>(__VA_ARGS__)   \
     : padded_vd(vd) == 8  ? launch_slice<PD_, 8>(__VA_ARGS__)  \
     : padded_vd(vd) == 12 ? launch_slice<PD_, 12>(__VA_ARGS__) \
     : padded_vd(vd) == 16 ? launch_slice<PD_, 16>(__VA_ARGS__) \
     : padded_vd(vd) == 20 ? launch_slice<PD_, 20>(__VA_ARGS__) \
     : padded_vd(vd) == 24 ? launch_slice<PD_, 24>(__VA_ARGS__) \
     : padded_vd(vd) == 28 ? launch_slice<PD_, 28>(__VA_ARGS__) \
     : padded_vd(vd) == 32 ? launch_slice<PD_, 32>(__VA_ARGS__) \
                           : launch_slice<PD_, 0>(__VA_ARGS__))

// Whether a bound is the worst case, which lattices of points with nothing in common need and fill.  Other bounds are 1.5 times the
// entries or more, of which a half at most are vertices, usually.
static bool worst_case(const Geom& g, int pd, const Layout& L) { return L.max_entries >= (u64)g.batch * (u64)g.n * (u64)(pd + 1); }
// Which calls take the kernels of small.cuh, by the bounds the host knows.  The index as far as its shared memory goes: 3074 entries
// 17.8 (one cluster on global memory) -> 9.4 us, 7017 entries 20.7 -> 17, as long as the three wide launches by then.  With pd 4 and 5 an
// entry takes 16 bytes beside the table, which is left 2.1 slots an entry at 9216 of them and 1.5 at 10240, too few: us a call, small / wide,
// all of the bound vertices, pd 4, 9200 50 / 44, 10200 71 / 44, pd 5 52 / 47 and 66 / 47 (few of them: 24 / 27); other pd 41 / 40 to 93 / 87 at
// 10200.  So bounds of the worst case end there.
static bool small_index(const Geom& g, int pd, const Layout& L) {
    return L.max_entries <= (worst_case(g, pd, L) && (pd == 4 || pd == 5) ? 9216u : SMALL_MAX_ENTRIES);
}
// A cluster for every 16 bytes of a row, as many as the GPU takes at once (two CTAs an SM while a thread has one vertex, else
// one), or twice as many of the small ones.  Six passes, us, wide (a pass a launch) / in one launch, by the bound: 4096, 1 float4 a row 15 /
// 7, 3 float4 14 / 9; 12000, 1 float4 15 / 12; 30000, 6 float4 15 / 14.6, and five launches less for the host, which such calls
// wait for: 2 x 100x100 x 21, forward + backward, 170 / 146 us.  That is with a third of the bound or less in vertices.  Bounds of the worst
// case may be all vertices, up to 32 k of them on eight SMs, and go on to two vertices a thread: us a call, two passes a launch / in one, 3
// channels, pd 4, 12 k vertices 45 / 47, 21 k 49 / 60; pd 8, 9 k 57 / 62, 18 k 58 / 75; pd 16, 10 k 83 / 92, 25 k 86 / 116; without a guide 24 k
// 31 / 42; few vertices, bounds of 9000 and 10000, pd 5 30 / 27, pd 4 30 / 26.6, pd 2 42 / 38.
constexpr int SMALL_PIECES = 4;   // vertices a thread of blur_small, at most
static bool small_blur(const Geom& g, int pd, const Layout& L, u32 vpr) {
    const u64 one_each = SMALL_CTAS * SMALL_THREADS;
    if (L.max_entries <= one_each) return vpr <= 64;
    const int pieces = worst_case(g, pd, L) ? 2 : SMALL_PIECES;
    return L.max_entries <= pieces * one_each && vpr <= 16;
}
// Where one lattice serves several items, the rows of a vertex lie together, and a cluster's 16 bytes of them far apart: up to eight
// float4 a vertex.  us a call, two passes a launch / all in one: 64x64x64 x 1 26 / 45, 16x128x128 x 1 26 / 34, 2x256x256 x 21 32 / 37.
constexpr u32 SMALL_SHARED = 8;
// A batch that is small as a whole, and would have its blur in one launch with a lattice of all items but not with one for them all: such a
// call waits for its launches, as long as the construction of all takes no longer than that of one, with a tile an SM or fewer.  us a
// call, a lattice each / one: 64x8x8 x 1 22 / 24, 4x64x64 x 21 23.8 / 25.7; with more tiles 64x32x32 x 1 28 / 24, 16x64x64 x 21 36 / 27.
static bool better_each(const Geom& g, int pd, const Layout& whole, u32 quads) {
    return g.num_tiles <= num_sms() && quads * (u32)g.batch > SMALL_SHARED && small_blur(g, pd, whole, quads);
}
// Two passes a launch (see blur_pair_rows), by what the bound says of the vertices.  us a call, a pass / two a launch: bounds
// of 393 k x 2 items, 115 k vertices (512x512 x 3 in double, forward + backward) 185 / 179; worst cases filled by vertices: 240 k
// 99.3 / 98.2, 470 k 142 / 144, 960 k 239 / 254.
static bool blur_in_pairs(const Geom& g, int pd, const Layout& L, u32 vpr) {
    return L.max_entries * vpr <= (worst_case(g, pd, L) ? PAIR_ITEMS_WORST : PAIR_ITEMS);
}
template <int PD, int KW, bool SHARED>
static int launch_small_index_as(Header* hdr, const Layout& L, const Key<KW>* list_keys, u32* list_ref, Key<KW>* vkeys,
                              const VertexInit& vinit, const ItemRows& rows, Watch watch, cudaStream_t st) {
    const u32 entries = (u32)L.max_entries;   // (times the items: no more than the call's bound)
    const size_t smem = SmallIndex<PD>::bytes(entries);
    PL_TRY((ensure_dynamic_smem<index_small<PD, KW, SHARED>>(smem)));
    // a thread for every axis and vertex, up to 64 CTAs, and for the entries and rows of all items, up to one CTA an SM
    const u64 of_items = SHARED ? ((u64)entries * rows.items + SMALL_THREADS - 1) / SMALL_THREADS : 0;
    const u32 ctas = std::max(std::max(8u, std::min(64u, (entries * (PD + 1) + SMALL_THREADS - 1) / SMALL_THREADS)),
                              (u32)std::min(of_items, (u64)num_sms()));
    PL_LAUNCH_AFTER(true, (index_small<PD, KW, SHARED>), ctas, SMALL_THREADS, smem, st, hdr, list_keys, list_ref, vkeys, vinit, rows,
            (u32)smem, watch);
    return PL_OK;
}
template <int PD, int KW>
static int launch_small_index(Header* hdr, const Layout& L, const Key<KW>* list_keys, u32* list_ref, Key<KW>* vkeys,
                              const VertexInit& vinit, const ItemRows& rows, Watch watch, cudaStream_t st) {
    if constexpr (PD <= MAX_SDIMS) {
        if (rows.items > 1) return launch_small_index_as<PD, KW, true>(hdr, L, list_keys, list_ref, vkeys, vinit, rows, watch, st);
    }
    return launch_small_index_as<PD, KW, false>(hdr, L, list_keys, list_ref, vkeys, vinit, rows, watch, st);
}
template <typename V, int PIECES>
static int launch_small_blur_as(const Header* hdr, const int* nbr, const Layout& L, V* v, u32 vpr, int axes, int reverse, cudaStream_t st) {
    const size_t smem = sizeof(V) * 2 * PIECES * SMALL_THREADS;
    PL_TRY((ensure_dynamic_smem<blur_small<V, PIECES>>(smem)));
    PL_LAUNCH_AFTER(true, (blur_small<V, PIECES>), SMALL_CTAS * vpr, SMALL_THREADS, smem, st, hdr, nbr, L.max_entries, v, vpr, axes, reverse);
    return PL_OK;
}
template <typename V>
static int launch_small_blur(const Header* hdr, const int* nbr, const Layout& L, V* v, u32 vpr, int axes, int reverse, cudaStream_t st) {
    const u64 pieces = (L.max_entries + SMALL_CTAS * SMALL_THREADS - 1) / (SMALL_CTAS * SMALL_THREADS);   // a thread
    return pieces <= 1   ? launch_small_blur_as<V, 1>(hdr, nbr, L, v, vpr, axes, reverse, st)
           : pieces <= 2 ? launch_small_blur_as<V, 2>(hdr, nbr, L, v, vpr, axes, reverse, st)
                         : launch_small_blur_as<V, SMALL_PIECES>(hdr, nbr, L, v, vpr, axes, reverse, st);
}

// The header's counters and, in calls that keep one, the sketch behind it.
static int clear_header_of(Header* hdr, int sketch_shift, const ClearTable& clear, cudaStream_t st) {
    const unsigned ctas = std::min(1u + clear.quads / 1024u, 2u * (unsigned)num_sms());
    // (the split of the build beside it, see launch_absmax; a microsecond of the host that small calls are better without)
    if (clear.quads > (1u << 16)) PL_TRY((ensure_dynamic_smem<clear_header>(16, true)));
    PL_LAUNCH((clear_header), ctas, 256, 0, st, hdr, (u32)((sketch_shift >= 0 ? HEADER_BYTES : sizeof(Header)) / 16), clear);
    PL_COUNT_LAUNCHES(1);
    return PL_OK;
}

// The deterministic mode's largest magnitude, beside the next kernel (see absmax_kernel).  Its CTAs use no shared memory, but are split as
// those of the tile kernels are: an SM takes CTAs of another split only when it is empty, and nothing overlapped.  Two CTAs an SM.
static int launch_absmax(const float* input, const Geom& g, int vd, Header* hdr, cudaStream_t st) {
    PL_TRY((ensure_dynamic_smem<absmax_kernel>(16, true)));
    PL_LAUNCH_AFTER(true, (absmax_kernel), num_sms() * 2, 256, 0, st, input, (u64)g.batch * g.n * (vd - 1), hdr);
    PL_COUNT_LAUNCHES(1);
    return PL_OK;
}

enum { PH_BUILD = 1, PH_APPLY = 2 };   // halves of a call: lattice structure / values through it

// KW: words of a key.
template <int PD, int KW>
static int run_filter(const Geom& call, float* output, const float* input, const float* positions,
                      const float* reference, int vd, int reverse, int mode, void* workspace,
                      const Layout& whole, cudaStream_t st, int phases = PH_BUILD | PH_APPLY) {
    constexpr int TP = Cfg<PD>::TP;
    // g, L: of the whole call; the lattice is that of `one`, within `share` of the bound (see one_for_all)
    Geom g = call, one;
    Layout share;
    const bool together = phases == (PH_BUILD | PH_APPLY) && !better_each(call, PD, whole, (u32)padded_vd(vd) / 4) && one_for_all(call,
            whole, PD, vd, one, share);
    if (together) {
        g.lattice_items = one.lattice_items;
        g.item_entries = one.item_entries;
    } else {
        one = call;
        share = whole;
    }
    const Layout& L = whole;
    const u32 items = (u32)one.lattice_items;
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    Header* hdr = reinterpret_cast<Header*>(ws);
    int2* tile_info = reinterpret_cast<int2*>(ws + L.tile_info);
    u16* rec = reinterpret_cast<u16*>(ws + L.rec);
    float* rec_w = reinterpret_cast<float*>(ws + L.rec_w);
    uint2* srec = reinterpret_cast<uint2*>(ws + L.srec);
    if (srec_words_of(PD) != Cfg<PD>::SREC) return PL_INTERNAL_ERROR;   // the layout and the kernels agree on the stride
    Key<KW>* list_keys = reinterpret_cast<Key<KW>*>(ws + L.list_keys);
    u32* list_ref = reinterpret_cast<u32*>(ws + L.list_ref);
    u32* vid = reinterpret_cast<u32*>(ws + L.vid);
    Key<KW>* vkeys = reinterpret_cast<Key<KW>*>(ws + L.vkeys);
    u64* table = reinterpret_cast<u64*>(ws + L.table);
    int* nbr = reinterpret_cast<int*>(ws + L.nbr);
    float* v0 = reinterpret_cast<float*>(ws + L.v0);
    float* v1 = reinterpret_cast<float*>(ws + L.v1);
    long long* v64 = (mode == PL_MODE_DETERMINISTIC) ? reinterpret_cast<long long*>(ws + L.v64) : nullptr;

    int sketch_shift = -1;   // no sketch
    cudaEvent_t* ev = g_stage_events;
    g_stage_events = nullptr;
    if (ev) PL_CUDA(cudaEventRecord(ev[0], st));
    Direct direct;
    bool use_direct = false, small = false, cleared = false;
    if (phases & PH_BUILD) {
        if constexpr (PD <= MAX_SDIMS) use_direct = make_direct(direct, call, PD, L);
        if (together) direct.slots = direct.cells;
        small = !use_direct && small_index(one, PD, share);
        const ClearTable clear = table_to_clear(use_direct ? &direct : nullptr, share, table, small, !Cfg<PD>::COMPACT);
        cleared = clear.table != nullptr;
        if (!use_direct && !small && !cleared) sketch_shift = sketch_shift_of(share.max_entries);
        PL_TRY(clear_header_of(hdr, sketch_shift, clear, st));
        if (v64 && (phases & PH_APPLY)) PL_TRY(launch_absmax(input, call, vd, hdr, st));
    }
    if (g.num_tiles == 0) return PL_OK;
    const Watch watch = (phases & PH_BUILD) ? take_watch(st) : Watch{nullptr, 0u};

    PL_TRY((ensure_dynamic_smem<build_tiles<PD, float, false, KW>>(Cfg<PD>::build_smem(false))));
    const int sms = num_sms();
    const int wide = sms * 8;
    int table_log2 = 0;
    while ((1ull << table_log2) < share.table_slots) table_log2++;

    // The insert overlaps clear_table only in regions of up to 64 MB of 8-byte slots (pd up to 5: 2^23 slots too, 128 MB, of
    // which the device uses what the vertices ask for): behind a clear_table that itself overlaps build_tiles it cost
    // calls with large tables 4-25 % (pd 16: 30 -> 37 ms)
    const bool small_table = L.index_words <= (1ull << 24);
    if (phases & PH_BUILD) {
        // what the insert overlaps: clear_table (see above), or the build itself
        const bool before_insert = cleared || small_table;
        // (beyond pd 8 the build has to wait for the header at its start, and launched beside it took 112 -> 128 us)
        constexpr bool beside_clear = !Cfg<PD>::COMPACT;
        // a lattice built to be applied later (no values in this call) also gets its splats sorted
        if (phases & PH_APPLY) {
            PL_LAUNCH_AFTER(beside_clear, (build_tiles<PD, float, false, KW>), tile_grid(one), TP, Cfg<PD>::build_smem(false), st, one,
                    positions, reference, hdr,
                                                                         tile_info, rec, rec_w, srec, list_keys,
                                                                                 (u32)share.max_entries, sketch_shift);
        } else {
            PL_TRY((ensure_dynamic_smem<build_tiles<PD, float, true, KW>>(Cfg<PD>::build_smem(true))));
            PL_LAUNCH_AFTER(beside_clear, (build_tiles<PD, float, true, KW>), tile_grid(g), TP, Cfg<PD>::build_smem(true), st, g, positions, reference, hdr,
                                                                        tile_info, rec, rec_w, srec, list_keys, (u32)L.max_entries, sketch_shift);
        }
        if (ev) PL_CUDA(cudaEventRecord(ev[1], st));
        // a new vertex's neighbour slots are initialised by the launch that creates it, its value row (when this call also
        // applies) by the link launch
        VertexInit vinit;
        vinit.nbr = nbr;
        vinit.max_entries = share.max_entries;
        vinit.pd = PD;
        ItemRows rows;
        rows.items = items;
        rows.stride = one.item_entries;
        rows.row_step = one.row_step;
        rows.item_step = one.row_step > 1 ? 1u : one.item_entries;
        rows.rows = (phases & PH_APPLY) ? (v64 ? reinterpret_cast<uint4*>(v64) : reinterpret_cast<uint4*>(v0)) : nullptr;
        rows.row_quads = (u32)padded_vd(vd) / (v64 ? 2u : 4u);
        // what the insert says of an entry and the link resolves: in a list that is not the items', whose entries come from it, all of them
        u32* owners = together ? vid + share.max_entries : list_ref;
        if constexpr (PD <= MAX_SDIMS) {
            if (use_direct) {
                u32* table32 = reinterpret_cast<u32*>(table);
                if (!cleared) PL_LAUNCH_AFTER(true, (clear_direct), wide, 256, 0, st, hdr, table32, direct.slots);
                PL_LAUNCH_AFTER(before_insert, (insert_direct<PD>), wide, 256, 0, st, hdr, direct, table32, list_keys, owners, vid, vkeys, vinit);
                PL_LAUNCH_AFTER(true, (link_neighbours_direct<PD>), wide, 256, 0, st, hdr, direct, table32, owners, list_ref, vid, vkeys, nbr,
                                                                 share.max_entries, rows, watch);
            }
        }
        PL_COUNT_LAUNCHES(small ? 2 : cleared ? 3 : 4);   // build_tiles and the launches of the index stage
        if (small) {
            PL_TRY((launch_small_index<PD, KW>(hdr, share, list_keys, list_ref, vkeys, vinit, rows, watch, st)));
        } else if (!use_direct) {
            auto hash_index = [&](auto keys_in_slots) -> int {
                constexpr bool KEYS = decltype(keys_in_slots)::value;
                if (!cleared) PL_LAUNCH_AFTER(true, (clear_table<KEYS>), wide, 256, 0, st, hdr, table, (u32)table_log2, sketch_shift);
                if constexpr (KEYS)
                    PL_LAUNCH_AFTER(before_insert, (insert_keys<PD>), wide, 256, 0, st, hdr, reinterpret_cast<KeySlot*>(table),
                            (u32)table_log2, list_keys, owners, vid, vkeys, vinit, cleared);
                else
                    PL_LAUNCH_AFTER(before_insert, (insert_entries<KW>), wide, 256, 0, st, hdr, table, (u32)table_log2, list_keys,
                            owners, vid, vkeys, vinit, cleared);
                PL_LAUNCH_AFTER(true, (link_neighbours<PD, KEYS, KW>), link_grid<PD>(wide, share.max_entries), 256, 0, st, hdr, table,
                        (u32)table_log2, owners, list_ref, vid, vkeys, nbr,
                                                          share.max_entries, rows, watch);
                return PL_OK;
            };
            if constexpr (Cfg<PD>::KEY_SLOTS) {
                if (L.key_slots) PL_TRY(hash_index(std::true_type{}));
                else PL_TRY(hash_index(std::false_type{}));
            } else {
                PL_TRY(hash_index(std::false_type{}));
            }
        }
        if (ev) PL_CUDA(cudaEventRecord(ev[2], st));
    } else {
        if (ev) { PL_CUDA(cudaEventRecord(ev[1], st)); }
        PL_LAUNCH_AFTER(true, (zero_rows), wide, 256, 0, st, hdr, v0, v64, padded_vd(vd));
        PL_COUNT_LAUNCHES(1);
        if (ev) { PL_CUDA(cudaEventRecord(ev[2], st)); }
    }
    if (!(phases & PH_APPLY)) {
        PL_CUDA(cudaGetLastError());
        return PL_OK;
    }
    // the blur passes (and the conversion of the fixed-point sums): on the rows of a vertex, or with a row of blocks for every item
    const u32 quads = (u32)padded_vd(vd) / 4, qpr = quads * one.row_step, apart = one.row_step > 1 ? 1u : items;
    const u64 item_v = (u64)one.item_entries * quads;
    auto blocks_of = [&](int blocks) { return dim3((unsigned)((blocks + (int)apart - 1) / (int)apart), apart); };
    int rc = PL_OK;
    if (v64) {
        if (vd > widest_vd_fixed(PD)) return PL_UNSUPPORTED_DIMS;
        if (!(phases & PH_BUILD)) PL_TRY(launch_absmax(input, call, vd, hdr, st));
        rc = (phases & PH_BUILD) ? launch_splat_fixed<PD, false>(g, input, hdr, tile_info, rec, rec_w, srec, list_ref, v64, vd, st)
                                 : launch_splat_fixed<PD, true>(g, input, hdr, tile_info, rec, rec_w, srec, list_ref, v64, vd, st);
        if (rc != PL_OK) return rc;
        PL_LAUNCH_AFTER(true, (convert_fixed), blocks_of(wide), 256, 0, st, hdr, v64, v0, qpr * 4, item_v * 4);
        PL_COUNT_LAUNCHES(1);   // convert_fixed (the splat itself is counted below)
    } else {
        rc = PL_SPLAT_FOR(PD, vd, g, input, hdr, tile_info, rec, rec_w, srec, !(phases & PH_BUILD), list_ref, v0, vd, st);
    }
    if (rc != PL_OK) return rc;
    PL_COUNT_LAUNCHES(1 + 1);   // splat, slice (the blur launches are counted where they are issued)
    if (ev) PL_CUDA(cudaEventRecord(ev[3], st));
    float* src = v0;
    float* dst = v1;
    const bool one_blur = apart == 1 && small_blur(one, PD, share, qpr) && (items == 1 || qpr <= SMALL_SHARED);
    if (one_blur) {
        PL_TRY(launch_small_blur(hdr, nbr, share, reinterpret_cast<float4*>(v0), qpr, PD + 1, reverse, st));
        PL_COUNT_LAUNCHES(1);
    } else if (blur_in_pairs(one, PD, share, quads * items)) {
        for (int step = 0; step <= PD; step += 2) {
            const int* nb = nbr + (size_t)(reverse ? PD - step : step) * share.max_entries * 2;
            const int* then = step == PD ? nullptr : nbr + (size_t)(reverse ? PD - step - 1 : step + 1) * share.max_entries * 2;
            PL_LAUNCH_AFTER(true, (blur_pair<float4>), blocks_of(sms * PAIR_CTAS), 256, 0, st, hdr, nb, then,
                    reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), qpr, item_v);
            std::swap(src, dst);
            PL_COUNT_LAUNCHES(1);
        }
    } else for (int step = 0; step <= PD; step++) {
        const int axis = reverse ? PD - step : step;
        const int* nb = nbr + (size_t)axis * share.max_entries * 2;
        PL_LAUNCH_AFTER(true, (blur_axis<float4>), blocks_of(wide), 256, 0, st, hdr, nb, reinterpret_cast<const float4*>(src),
                reinterpret_cast<float4*>(dst), qpr, item_v);
        float* tmp = src; src = dst; dst = tmp;
        PL_COUNT_LAUNCHES(1);
    }
    if (ev) PL_CUDA(cudaEventRecord(ev[4], st));
    rc = PL_SLICE_FOR(PD, vd, g, output, hdr, tile_info, rec, rec_w, list_ref, src, vd, watch, slice_overlap(g, one_blur), st);
    if (rc != PL_OK) return rc;
    if (ev) PL_CUDA(cudaEventRecord(ev[5], st));
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

// T = double: the same structure kernels, then splat, blur and slice over rows of doubles.
template <int PD>
static int run_filter_f64(const Geom& g, double* output, const double* input, const double* positions,
                          const double* reference, int vd, int reverse, void* workspace, const Layout& L,
                          cudaStream_t st) {
    constexpr int KW = Cfg<PD>::KW, TP = Cfg<PD>::TP;
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    Header* hdr = reinterpret_cast<Header*>(ws);
    int2* tile_info = reinterpret_cast<int2*>(ws + L.tile_info);
    u16* rec = reinterpret_cast<u16*>(ws + L.rec);
    double* rec_w = reinterpret_cast<double*>(ws + L.rec_w);
    Key<KW>* list_keys = reinterpret_cast<Key<KW>*>(ws + L.list_keys);
    u32* list_ref = reinterpret_cast<u32*>(ws + L.list_ref);
    u32* vid = reinterpret_cast<u32*>(ws + L.vid);
    Key<KW>* vkeys = reinterpret_cast<Key<KW>*>(ws + L.vkeys);
    u64* table = reinterpret_cast<u64*>(ws + L.table);
    int* nbr = reinterpret_cast<int*>(ws + L.nbr);
    double* v0 = reinterpret_cast<double*>(ws + L.v0);
    double* v1 = reinterpret_cast<double*>(ws + L.v1);

    // spatial-only calls index their vertices directly, as the float calls do (the key bounds hold for
    // either arithmetic: the margin is far wider than any rounding)
    Direct direct;
    bool use_direct = false;
    if constexpr (PD <= MAX_SDIMS) use_direct = make_direct(direct, g, PD, L);
    const bool small = !use_direct && small_index(g, PD, L);
    const ClearTable clear = table_to_clear(use_direct ? &direct : nullptr, L, table, small, !Cfg<PD>::COMPACT);
    const bool cleared = clear.table != nullptr;
    const int sketch_shift = use_direct || small || cleared ? -1 : sketch_shift_of(L.max_entries);
    PL_TRY(clear_header_of(hdr, sketch_shift, clear, st));
    if (g.num_tiles == 0) return PL_OK;
    const Watch watch = take_watch(st);
    PL_TRY((ensure_dynamic_smem<build_tiles<PD, double>>(Cfg<PD>::build_smem(false))));
    const size_t splat_smem = Splat64<PD>::bytes(vd);
    PL_TRY((ensure_dynamic_smem<splat_tiles_f64<PD>>(splat_smem)));
    const int wide = num_sms() * 8;
    int table_log2 = 0;
    while ((1ull << table_log2) < L.table_slots) table_log2++;
    const int vp = padded_vd_f64(vd);
    const bool small_table = L.index_words <= (1ull << 24);   // (as for float)
    const bool before_insert = cleared || small_table;

    PL_LAUNCH_AFTER(!Cfg<PD>::COMPACT, (build_tiles<PD, double>), tile_grid(g), TP, Cfg<PD>::build_smem(false), st, g, positions,
            reference, hdr, tile_info, rec, rec_w, static_cast<uint2*>(nullptr), list_keys, (u32)L.max_entries, sketch_shift);
    u32* table32 = reinterpret_cast<u32*>(table);
    VertexInit vinit;
    vinit.nbr = nbr;
    vinit.max_entries = L.max_entries;
    vinit.pd = PD;
    const ItemRows rows = {1u, 0u, 1u, 0u, reinterpret_cast<uint4*>(v0), (u32)vp / 2};   // rows of vp doubles
    if constexpr (PD <= MAX_SDIMS) {
        if (use_direct) {
            if (!cleared) PL_LAUNCH_AFTER(true, (clear_direct), wide, 256, 0, st, hdr, table32, direct.slots);
            PL_LAUNCH_AFTER(before_insert, (insert_direct<PD>), wide, 256, 0, st, hdr, direct, table32, list_keys, list_ref, vid, vkeys, vinit);
            PL_LAUNCH_AFTER(true, (link_neighbours_direct<PD>), wide, 256, 0, st, hdr, direct, table32, list_ref, list_ref, vid, vkeys, nbr,
                                                             L.max_entries, rows, watch);
        }
    }
    if (small) {
        PL_TRY((launch_small_index<PD, KW>(hdr, L, list_keys, list_ref, vkeys, vinit, rows, watch, st)));
    } else if (!use_direct) {
        if (!cleared) PL_LAUNCH_AFTER(true, (clear_table<Cfg<PD>::KEY_SLOTS>), wide, 256, 0, st, hdr, table, (u32)table_log2, sketch_shift);
        if constexpr (Cfg<PD>::KEY_SLOTS)
            PL_LAUNCH_AFTER(before_insert, (insert_keys<PD>), wide, 256, 0, st, hdr, reinterpret_cast<KeySlot*>(table), (u32)table_log2, list_keys, list_ref, vid, vkeys, vinit, cleared);
        else
            PL_LAUNCH_AFTER(before_insert, (insert_entries<KW>), wide, 256, 0, st, hdr, table, (u32)table_log2, list_keys, list_ref, vid, vkeys, vinit, cleared);
        PL_LAUNCH_AFTER(true, (link_neighbours<PD, Cfg<PD>::KEY_SLOTS>), link_grid<PD>(wide, L.max_entries), 256, 0, st, hdr, table,
                (u32)table_log2, list_ref, list_ref, vid, vkeys, nbr, L.max_entries,
                                                  rows, watch);
    }
    PL_LAUNCH_AFTER(true, (splat_tiles_f64<PD>), tile_grid(g), TP, splat_smem, st, g, input, hdr, tile_info, rec, rec_w,
                                                                      list_ref, v0, vd);
    double* src = v0;
    double* dst = v1;
    const bool one_blur = small_blur(g, PD, L, (u32)vp / 2), pairs = blur_in_pairs(g, PD, L, (u32)vp / 2);
    if (one_blur) {
        PL_TRY(launch_small_blur(hdr, nbr, L, reinterpret_cast<double2*>(v0), (u32)vp / 2, PD + 1, reverse, st));
    } else if (pairs) {
        for (int step = 0; step <= PD; step += 2) {
            const int* nb = nbr + (size_t)(reverse ? PD - step : step) * L.max_entries * 2;
            const int* then = step == PD ? nullptr : nbr + (size_t)(reverse ? PD - step - 1 : step + 1) * L.max_entries * 2;
            PL_LAUNCH_AFTER(true, (blur_pair<double2>), num_sms() * PAIR_CTAS, 256, 0, st, hdr, nb, then,
                    reinterpret_cast<const double2*>(src), reinterpret_cast<double2*>(dst), (u32)vp / 2, (u64)0);
            std::swap(src, dst);
        }
    } else for (int step = 0; step <= PD; step++) {
        const int axis = reverse ? PD - step : step;
        PL_LAUNCH_AFTER(true, (blur_axis<double2>), wide, 256, 0, st, hdr, nbr + (size_t)axis * L.max_entries * 2,
                reinterpret_cast<const double2*>(src), reinterpret_cast<double2*>(dst), (u32)vp / 2, (u64)0);
        double* tmp = src; src = dst; dst = tmp;
    }
    PL_LAUNCH_AFTER(vd <= 4 || slice_overlap(g, one_blur), (slice_tiles_f64<PD>), tile_grid(g), TP, 0, st, g, output, hdr, tile_info,
            rec, rec_w, list_ref, src, vd, watch);
    PL_COUNT_LAUNCHES((small ? 2 : cleared ? 3 : 4) + 1 + (one_blur ? 1 : pairs ? PD / 2 + 1 : PD + 1) + 1);   // build and index; splat; blur; slice
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

// crf_update, or without messages (crf.cuh) the start of an inference.
static int launch_crf_update(float* q_out, const float* unaries, const float* q_bilateral, const float* q_spatial,
                             const float* compatibility, float bilateral_weight, float spatial_weight, int64_t n_points,
                             int n_labels, cudaStream_t st) {
    const int tpb = n_labels <= 32 ? 256 : 128;
    const size_t smem = crf_smem_bytes(tpb, n_labels);
    const long long blocks = (n_points + tpb - 1) / tpb;
    if (blocks > 0x7FFFFFFFll) return PL_INVALID_ARGUMENT;
#define PL_CRF_LAUNCH(TPB, LT)                                                                                   \
    do {                                                                                                         \
        PL_TRY((ensure_dynamic_smem<crf_update<TPB, LT>>(smem)));                                                \
        crf_update<TPB, LT><<<(unsigned)blocks, TPB, smem, st>>>(q_out, unaries, q_bilateral, q_spatial,         \
                                                                 compatibility, bilateral_weight, spatial_weight, \
                                                                 n_points, n_labels);                            \
    } while (0)
    // Potts model at the label count of the benchmark's CRF (20 classes + background): rows in registers
    if (n_labels == 21 && !compatibility) PL_CRF_LAUNCH(256, 21);
    else if (n_labels <= 32) PL_CRF_LAUNCH(256, 0);
    else PL_CRF_LAUNCH(128, 0);
    PL_COUNT_LAUNCHES(1);
#undef PL_CRF_LAUNCH
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

// Whose keys hold no item (float calls; see Cfg::KW_ALONE): the same for whoever reads the workspace later.
static bool batch_of_one(const Geom& g) { return g.batch == 1; }

// A mean-field step through two kept lattices (crf.cuh).
static LatticeRows lattice_rows(void* workspace, const Layout& L) {
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    LatticeRows l;
    l.hdr = reinterpret_cast<Header*>(ws);
    l.tile_info = reinterpret_cast<const int2*>(ws + L.tile_info);
    l.rec = reinterpret_cast<const u16*>(ws + L.rec);
    l.rec_w = reinterpret_cast<const float*>(ws + L.rec_w);
    l.srec = reinterpret_cast<const uint2*>(ws + L.srec);
    l.list_ref = reinterpret_cast<const u32*>(ws + L.list_ref);
    l.nbr = reinterpret_cast<const int*>(ws + L.nbr);
    l.max_entries = L.max_entries;
    l.v0 = reinterpret_cast<float*>(ws + L.v0);
    l.v1 = reinterpret_cast<float*>(ws + L.v1);
    return l;
}
template <int PDA, int PDS, int VD>
static int launch_crf_splat(const Geom& g, const float* q, const LatticeRows& a, const LatticeRows& s, int vd, cudaStream_t st) {
    const size_t smem = std::max(SplatRows<PDA, VD, true>::bytes(vd), SplatRows<PDS, VD, true>::bytes(vd));
    PL_TRY((ensure_dynamic_smem<crf_splat<PDA, PDS, VD>>(smem, true)));
    dim3 grid = tile_grid(g);
    (g.grid3 ? grid.z : grid.x) *= 2;
    PL_LAUNCH_AFTER(true, (crf_splat<PDA, PDS, VD>), grid, Cfg<PDA>::TP, smem, st, g, q, a, s, vd, bulk_staging_ok(g, q, vd) ? 1 : 0);
    return PL_OK;
}
template <int PDA, int PDS, int VP, int CT = 0>
static int launch_crf_slices(const Geom& g, float* q_out, const float* unaries, const LatticeRows& a, const LatticeRows& s,
                             const float* va, const float* vs, float wa, float ws, int labels, bool blurred_small, cudaStream_t st) {
    const size_t smem = CrfSlices<PDA, PDS, VP>::bytes(labels);
    PL_TRY((ensure_dynamic_smem<crf_slices<PDA, PDS, VP, CT>>(smem)));
    // (an even number of labels is spread to an odd stride, which a bulk copy cannot do)
    const bool bulk_in = (labels & 1) && bulk_rows_ok(g, unaries, labels), bulk_out = bulk_rows_ok(g, q_out, labels);
    PL_LAUNCH_AFTER(slice_overlap(g, blurred_small), (crf_slices<PDA, PDS, VP, CT>), tile_grid(g), Cfg<PDA>::TP, smem, st, g, q_out, unaries, a, s, va, vs, wa, ws, labels, bulk_in ? 1 : 0, bulk_out ? 1 : 0);
    return PL_OK;
}
// Pass by pass both lattices in one launch, as long as their rows may stay in L2 together: by the bounds, in pieces of 16 bytes.  us a step,
// together / one after the other: 375x500 x 21 (2.5 M) 66.3 / 71.5; 2 x 500x640 x 21 (9 M) 152.5 / 157.6; 4 x 512x512 x 21 (14 M) 265 / 271; 4 x
// 512x512 x 5 of noisy images (19 M) 208 / 212; 8 x 512x512 x 21 (26 M) 497 / 498; of noisy ones 2 x 512x512 x 21 (28 M) 468 / 450, 8 x
// 512x512 x 12 (45 M) 920 / 866, 2000x3000 x 10 (75 M and more) 2051 / 1869, 8 x 512x512 x 21 (113 M) 2076 / 1872.
constexpr u64 CRF_TOGETHER = 20000000;
template <int PDA, int PDS>
static int run_crf_step(const Geom& g, float* q_out, const float* q, const float* unaries, float wa, float wsp, int labels,
                        void* ws_a, const Layout& LA, void* ws_s, const Layout& LS, cudaStream_t st) {
    const LatticeRows a = lattice_rows(ws_a, LA), s = lattice_rows(ws_s, LS);
    const int vd = labels + 1, vp = padded_vd(vd), wide = num_sms() * 8;
    const u32 quads = (u32)vp / 4;
    PL_LAUNCH_AFTER(true, (crf_zero_rows), dim3(wide / 2, 2), 256, 0, st, a, s, quads);
    PL_TRY((vd == 22 ? launch_crf_splat<PDA, PDS, 22>(g, q, a, s, vd, st) : launch_crf_splat<PDA, PDS, 0>(g, q, a, s, vd, st)));
    // small lattices have all their passes in one launch each; else a launch a pass, both as long as S has some left
    const bool small_a = small_blur(g, PDA, LA, quads), small_s = small_blur(g, PDS, LS, quads);
    const float *va = a.v0, *vs = s.v0;
    int launches = 3;
    if (small_s) {
        PL_TRY(launch_small_blur(s.hdr, s.nbr, LS, reinterpret_cast<float4*>(s.v0), quads, PDS + 1, 0, st));
        launches++;
    }
    if (small_a) {
        PL_TRY(launch_small_blur(a.hdr, a.nbr, LA, reinterpret_cast<float4*>(a.v0), quads, PDA + 1, 0, st));
        launches++;
    }
    const bool pairs = blur_in_pairs(g, PDA, LA, quads) && blur_in_pairs(g, PDS, LS, quads);
    for (int pair = 0; pairs && pair <= std::max(PDA, PDS) / 2; pair++) {
        const bool pass_a = !small_a && 2 * pair <= PDA, pass_s = !small_s && 2 * pair <= PDS, both = pass_a && pass_s;
        if (!pass_a && !pass_s) continue;
        PL_LAUNCH_AFTER(true, (crf_blur_pair<PDA, PDS>), dim3(num_sms() * PAIR_CTAS / (both ? 2 : 1), both ? 2 : 1), 256, 0, st, a, s,
                both ? 0 : pass_a ? 1 : 2, pair, quads);
        launches++;
        if (pass_a) va = (pair & 1) ? a.v0 : a.v1;
        if (pass_s) vs = (pair & 1) ? s.v0 : s.v1;
    }
    // a pass of one lattice, from v0 to v1 in even passes
    struct Pass {
        const int* nbr;
        const float4* src;
        float4* dst;
    };
    auto pass_of = [](const LatticeRows& l, int step) {
        float4* const v[2] = {reinterpret_cast<float4*>(l.v0), reinterpret_cast<float4*>(l.v1)};
        return Pass{l.nbr + 2 * (u64)step * l.max_entries, v[step & 1], v[1 - (step & 1)]};
    };
    auto rest_of = [&](const LatticeRows& l, int step, int pd, const float*& v) -> int {   // from pass `step` on
        for (; step <= pd; step++) {
            const Pass p = pass_of(l, step);
            PL_LAUNCH_AFTER(true, (blur_axis<float4>), wide, 256, 0, st, l.hdr, p.nbr, p.src, p.dst, quads, (u64)0);
            launches++;
            v = reinterpret_cast<const float*>(p.dst);
        }
        return PL_OK;
    };
    if (!pairs) {
        int step = 0;
        if (!small_a && !small_s && (LA.max_entries + LS.max_entries) * quads <= CRF_TOGETHER) {
            for (; step <= std::min(PDA, PDS); step++) {
                const Pass p = pass_of(a, step), q2 = pass_of(s, step);
                PL_LAUNCH_AFTER(true, (crf_blur), dim3(wide / 2, 2), 256, 0, st, a.hdr, p.nbr, p.src, p.dst, s.hdr, q2.nbr, q2.src, q2.dst, quads);
                launches++;
                va = reinterpret_cast<const float*>(p.dst);
                vs = reinterpret_cast<const float*>(q2.dst);
            }
        }
        if (!small_a) PL_TRY(rest_of(a, step, PDA, va));
        if (!small_s) PL_TRY(rest_of(s, step, PDS, vs));
    }
    PL_COUNT_LAUNCHES(launches);
#define PL_CRF_SLICES(VP_, ...) launch_crf_slices<PDA, PDS, VP_, ##__VA_ARGS__>(g, q_out, unaries, a, s, va, vs, wa, wsp, labels, small_a && small_s, st)
    PL_TRY((labels == 21 ? PL_CRF_SLICES(24, 21)
            : vp == 8    ? PL_CRF_SLICES(8)
            : vp == 12   ? PL_CRF_SLICES(12)
            : vp == 16   ? PL_CRF_SLICES(16)
            : vp == 20   ? PL_CRF_SLICES(20)
            : vp == 24   ? PL_CRF_SLICES(24)
            : vp == 28   ? PL_CRF_SLICES(28)
                         : PL_CRF_SLICES(32)));
#undef PL_CRF_SLICES
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

template <int PD, typename R, int KW>
static int run_export(const Geom& g, const R* positions, const R* reference, const void* workspace,
                      const Layout& L, long long max_vertices, int16_t* vertex_keys,
                      int32_t* vertex_item, int32_t* pixel_vertex, R* pixel_weight,
                      cudaStream_t st) {
    constexpr int TP = Cfg<PD>::TP;
    const unsigned char* ws = static_cast<const unsigned char*>(workspace);
    const Header* hdr = reinterpret_cast<const Header*>(ws);
    if (g.num_tiles == 0) return PL_OK;
    if (pixel_vertex || pixel_weight)
        export_points<PD, R><<<tile_grid(g), TP, 0, st>>>(
            g, hdr, reinterpret_cast<const int2*>(ws + L.tile_info), reinterpret_cast<const u16*>(ws + L.rec),
            reinterpret_cast<const R*>(ws + L.rec_w), reinterpret_cast<const u32*>(ws + L.list_ref),
            pixel_vertex, pixel_weight);
    if (vertex_keys || vertex_item)
        export_vertices<PD, KW><<<num_sms() * 4, 256, 0, st>>>(
            hdr, reinterpret_cast<const Key<KW>*>(ws + L.vkeys), max_vertices, vertex_keys, vertex_item);
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

#define PL_DISPATCH_PD(pd, CALL)            \
    switch (pd) {                           \
        case 1: return CALL(1);             \
        case 2: return CALL(2);             \
        case 3: return CALL(3);             \
        case 4: return CALL(4);             \
        case 5: return CALL(5);             \
        case 6: return CALL(6);             \
        case 7: return CALL(7);             \
        case 8: return CALL(8);             \
        case 16: return CALL(16);           \
        default: return PL_UNSUPPORTED_DIMS; \
    }

static int filter_common(const Geom& g, float* output, const float* input, const float* positions,
                         const float* reference, int pd, int vd, int reverse, void* workspace,
                         size_t workspace_bytes, int64_t max_entries, int mode, cudaStream_t st,
                         int phases = PH_BUILD | PH_APPLY, bool with_sorted = true) {
    if (mode != PL_MODE_ATOMIC && mode != PL_MODE_DETERMINISTIC) return PL_INVALID_ARGUMENT;
    Layout L;
    int rc = make_layout(L, g, pd, vd, max_entries, 4, mode == PL_MODE_DETERMINISTIC, with_sorted);
    if (rc != PL_OK) return rc;
    if (workspace_bytes < L.total) return PL_WORKSPACE_TOO_SMALL;
#define CALL(P) (batch_of_one(g) ? run_filter<P, Cfg<P>::KW_ALONE> : run_filter<P, Cfg<P>::KW>)(g, output, input, positions, reference, vd, reverse, mode, workspace, L, st, phases)
    PL_DISPATCH_PD(pd, CALL)
#undef CALL
}

// Scratch of pl_lattice_filter_f32_noalloc: lives in the library image, one copy on every GPU that
// loads the library, until the process exits.  In host code the array's name is only a handle; the
// device address comes from cudaGetSymbolAddress, once per device, with that device current.
static __device__ __align__(256) unsigned char g_static_scratch[PL_STATIC_SCRATCH_BYTES];
static void* g_static_scratch_addr[MAX_DEVICES] = {nullptr};
static std::mutex g_static_scratch_mutex;

static int static_scratch_of_current_device(void** out) {
    int dev = -1;
    PL_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return PL_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (!g_static_scratch_addr[dev]) {
        void* addr = nullptr;
        PL_CUDA(cudaGetSymbolAddress(&addr, g_static_scratch));
        g_static_scratch_addr[dev] = addr;
    }
    *out = g_static_scratch_addr[dev];
    return PL_OK;
}

}  // namespace pl

using namespace pl;

extern "C" {

int pl_supported(int pd, int vd) { return pd_supported(pd) && vd >= 2 && vd <= 4096 ? 1 : 0; }

const char* pl_strerror(int status) {
    switch (status) {
        case PL_OK: return "ok";
        case PL_INVALID_ARGUMENT: return "invalid argument";
        case PL_UNSUPPORTED_DIMS: return "unsupported (pd, vd)";
        case PL_WORKSPACE_TOO_SMALL: return "workspace too small";
        case PL_CAPACITY_EXCEEDED: return "lattice entries exceed max_entries";
        case PL_CUDA_ERROR: return "CUDA error";
        case PL_INTERNAL_ERROR: return "internal error (bounded device loop gave up)";
    }
    return "unknown status";
}

const char* pl_last_cuda_error(void) { return g_cuda_error; }

int pl_workspace_bytes(int batch, int n, int pd, int vd, int n_spatial_dims, const int* spatial_dims,
                       int64_t max_entries, int mode, size_t* bytes) {
    if (!bytes || batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (mode != PL_MODE_ATOMIC && mode != PL_MODE_DETERMINISTIC) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    Geom g;
    int rc;
    if (spatial_dims) {
        if (n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || n_spatial_dims > pd) return PL_INVALID_ARGUMENT;
        long long prod = 1;
        for (int i = 0; i < n_spatial_dims; i++) prod *= spatial_dims[i];
        if (prod != n) return PL_INVALID_ARGUMENT;
        rc = make_geom(g, batch, n, pd, n_spatial_dims, spatial_dims, pd - n_spatial_dims, 1.f, 1.f, false);
    } else {
        int one = n;
        rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    }
    if (rc != PL_OK) return rc;
    Layout L;
    rc = make_layout(L, g, pd, vd, max_entries, 4, mode == PL_MODE_DETERMINISTIC);
    if (rc != PL_OK) return rc;
    *bytes = L.total;
    return PL_OK;
}

int pl_compute_positions_f32(const float* reference, float* positions, int n,
                             int n_reference_channels, int n_spatial_dims, const int* spatial_dims,
                             float spatial_std, float feature_std, void* stream) {
    if (!positions || n < 0 || n_spatial_dims < 0 || n_spatial_dims > MAX_SDIMS ||
        n_reference_channels < 0 || (n_reference_channels > 0 && !reference) ||
        (n_spatial_dims > 0 && !spatial_dims))
        return PL_INVALID_ARGUMENT;
    if (n == 0) return PL_OK;
    Geom g;
    memset(&g, 0, sizeof(g));
    for (int i = 0; i < n_spatial_dims; i++) g.sdims[i] = spatial_dims[i];
    g.spatial_std = spatial_std;
    g.feature_std = feature_std;
    positions_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        reference, positions, n, n_reference_channels, n_spatial_dims, g);
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

int pl_filter_f32(float* output, const float* input, const float* positions, int batch, int n,
                  int pd, int vd, int reverse, void* workspace, size_t workspace_bytes,
                  int64_t max_entries, int mode, void* stream) {
    WatchScope this_call;
    if (batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || !positions || !workspace) return PL_INVALID_ARGUMENT;
    Geom g;
    int one = n;
    int rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    if (rc != PL_OK) return rc;
    return filter_common(g, output, input, positions, nullptr, pd, vd, reverse, workspace,
                         workspace_bytes, max_entries, mode, (cudaStream_t)stream);
}

static int op_geom(Geom& g, int batch, int n_spatial_dims, const int* spatial_dims,
                   int n_reference_channels, int bilateral, float theta_alpha, float theta_beta,
                   float theta_gamma, int* pd_out, int* n_out) {
    if (batch < 0 || batch > 65535 || n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || !spatial_dims ||
        n_reference_channels < 0)
        return PL_INVALID_ARGUMENT;
    long long n = 1;
    for (int i = 0; i < n_spatial_dims; i++) {
        if (spatial_dims[i] < 0) return PL_INVALID_ARGUMENT;
        n *= spatial_dims[i];
        if (n > 0x7FFFFFFFll) return PL_INVALID_ARGUMENT;
    }
    // src/LatticeFilterKernel.cpp:131-142
    const int R = bilateral ? n_reference_channels : 0;
    const int pd = n_spatial_dims + R;
    const float spatial_std = bilateral ? theta_alpha : theta_gamma;
    const float feature_std = bilateral ? theta_beta : -1.f;
    *pd_out = pd;
    *n_out = (int)n;
    if (!pd_supported(pd)) return PL_UNSUPPORTED_DIMS;
    return make_geom(g, batch, (int)n, pd, n_spatial_dims, spatial_dims, R, spatial_std, feature_std, false);
}

int pl_lattice_filter_f32(float* output, const float* input, const float* reference, int batch,
                          int n_spatial_dims, const int* spatial_dims, int n_input_channels,
                          int n_reference_channels, int bilateral, float theta_alpha,
                          float theta_beta, float theta_gamma, int reverse, void* workspace,
                          size_t workspace_bytes, int64_t max_entries, int mode, void* stream) {
    WatchScope this_call;
    if (n_input_channels < 1) return PL_INVALID_ARGUMENT;
    Geom g;
    int pd = 0, n = 0;
    int rc = op_geom(g, batch, n_spatial_dims, spatial_dims, n_reference_channels, bilateral,
                     theta_alpha, theta_beta, theta_gamma, &pd, &n);
    if (rc != PL_OK) return rc;
    const int vd = n_input_channels + 1;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || !workspace || (g.R > 0 && !reference)) return PL_INVALID_ARGUMENT;
    return filter_common(g, output, input, nullptr, reference, pd, vd, reverse, workspace,
                         workspace_bytes, max_entries, mode, (cudaStream_t)stream);
}

int pl_lattice_filter_f32_noalloc(float* output, const float* input, const float* reference, int batch,
                                  int n_spatial_dims, const int* spatial_dims, int n_input_channels,
                                  int n_reference_channels, int bilateral, float theta_alpha,
                                  float theta_beta, float theta_gamma, int reverse, int64_t max_entries,
                                  void* stream) {
    WatchScope this_call;
    if (n_input_channels < 1) return PL_INVALID_ARGUMENT;
    Geom g;
    int pd = 0, n = 0;
    int rc = op_geom(g, batch, n_spatial_dims, spatial_dims, n_reference_channels, bilateral, theta_alpha,
                     theta_beta, theta_gamma, &pd, &n);
    if (rc != PL_OK) return rc;
    const int vd = n_input_channels + 1;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || (g.R > 0 && !reference)) return PL_INVALID_ARGUMENT;
    // Sizes beyond the built-in scratch are refused before anything is launched.  The scratch has no room for sorted
    // splats, which a lattice used once does not keep.
    Layout L;
    rc = make_layout(L, g, pd, vd, max_entries, 4, false, false);
    if (rc != PL_OK) return rc;
    if (L.total > (size_t)PL_STATIC_SCRATCH_BYTES) {
        snprintf(g_cuda_error, sizeof(g_cuda_error),
                 "pl_lattice_filter_f32_noalloc: this call needs %zu bytes of scratch, the built-in scratch holds %zu",
                 L.total, (size_t)PL_STATIC_SCRATCH_BYTES);
        return PL_WORKSPACE_TOO_SMALL;
    }
    void* scratch = nullptr;
    rc = static_scratch_of_current_device(&scratch);   // first call on a device: looks the address up
    if (rc != PL_OK) return rc;
    // the call itself zeroes the counters it needs (the header and, in calls that keep one, the sketch behind it) and
    // the value rows it sums into; everything else in the scratch is written before it is read
    return filter_common(g, output, input, nullptr, reference, pd, vd, reverse, scratch,
                         (size_t)PL_STATIC_SCRATCH_BYTES, max_entries, PL_MODE_ATOMIC, (cudaStream_t)stream,
                         PH_BUILD | PH_APPLY, false);
}

int pl_lattice_build_f32(const float* reference, int batch, int n_spatial_dims, const int* spatial_dims,
                         int n_reference_channels, int bilateral, float theta_alpha, float theta_beta,
                         float theta_gamma, int max_value_dim, void* workspace, size_t workspace_bytes,
                         int64_t max_entries, void* stream) {
    WatchScope this_call;
    Geom g;
    int pd = 0, n = 0;
    int rc = op_geom(g, batch, n_spatial_dims, spatial_dims, n_reference_channels, bilateral, theta_alpha,
                     theta_beta, theta_gamma, &pd, &n);
    if (rc != PL_OK) return rc;
    if (!pl_supported(pd, max_value_dim)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!workspace || (g.R > 0 && !reference)) return PL_INVALID_ARGUMENT;
    return filter_common(g, nullptr, nullptr, nullptr, reference, pd, max_value_dim, 0, workspace, workspace_bytes,
                         max_entries, PL_MODE_ATOMIC, (cudaStream_t)stream, PH_BUILD);
}

int pl_lattice_build_positions_f32(const float* positions, int batch, int n, int pd, int max_value_dim,
                                   void* workspace, size_t workspace_bytes, int64_t max_entries, void* stream) {
    WatchScope this_call;
    if (batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, max_value_dim)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!positions || !workspace) return PL_INVALID_ARGUMENT;
    Geom g;
    int one = n;
    int rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    if (rc != PL_OK) return rc;
    return filter_common(g, nullptr, nullptr, positions, nullptr, pd, max_value_dim, 0, workspace, workspace_bytes,
                         max_entries, PL_MODE_ATOMIC, (cudaStream_t)stream, PH_BUILD);
}

int pl_lattice_apply_f32(float* output, const float* input, int n_input_channels, int reverse, int mode, int batch,
                         int n, int pd, int n_spatial_dims, const int* spatial_dims, void* workspace,
                         size_t workspace_bytes, int64_t max_entries, void* stream) {
    if (n_input_channels < 1 || batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    const int vd = n_input_channels + 1;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || !workspace) return PL_INVALID_ARGUMENT;
    Geom g;
    int rc;
    if (spatial_dims) {
        if (n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || n_spatial_dims > pd) return PL_INVALID_ARGUMENT;
        long long prod = 1;
        for (int i = 0; i < n_spatial_dims; i++) prod *= spatial_dims[i];
        if (prod != n) return PL_INVALID_ARGUMENT;
        rc = make_geom(g, batch, n, pd, n_spatial_dims, spatial_dims, pd - n_spatial_dims, 1.f, 1.f, false);
    } else {
        int one = n;
        rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    }
    if (rc != PL_OK) return rc;
    return filter_common(g, output, input, nullptr, nullptr, pd, vd, reverse, workspace, workspace_bytes,
                         max_entries, mode, (cudaStream_t)stream, PH_APPLY);
}

// ---------------------------------------------------------------------------------------------
// T = double
// ---------------------------------------------------------------------------------------------
static int geom_for_workspace(Geom& g, int batch, int n, int pd, int n_spatial_dims, const int* spatial_dims) {
    if (spatial_dims) {
        if (n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || n_spatial_dims > pd) return PL_INVALID_ARGUMENT;
        long long prod = 1;
        for (int i = 0; i < n_spatial_dims; i++) prod *= spatial_dims[i];
        if (prod != n) return PL_INVALID_ARGUMENT;
        return make_geom(g, batch, n, pd, n_spatial_dims, spatial_dims, pd - n_spatial_dims, 1.f, 1.f, false);
    }
    int one = n;
    return make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
}

int pl_workspace_bytes_f64(int batch, int n, int pd, int vd, int n_spatial_dims, const int* spatial_dims,
                           int64_t max_entries, size_t* bytes) {
    if (!bytes || batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    Geom g;
    int rc = geom_for_workspace(g, batch, n, pd, n_spatial_dims, spatial_dims);
    if (rc != PL_OK) return rc;
    Layout L;
    rc = make_layout(L, g, pd, vd, max_entries, 8);
    if (rc != PL_OK) return rc;
    *bytes = L.total;
    return PL_OK;
}

int pl_compute_positions_f64(const double* reference, double* positions, int n, int n_reference_channels,
                             int n_spatial_dims, const int* spatial_dims, double spatial_std,
                             double feature_std, void* stream) {
    if (!positions || n < 0 || n_spatial_dims < 0 || n_spatial_dims > MAX_SDIMS ||
        n_reference_channels < 0 || (n_reference_channels > 0 && !reference) ||
        (n_spatial_dims > 0 && !spatial_dims))
        return PL_INVALID_ARGUMENT;
    if (n == 0) return PL_OK;
    Geom g;
    memset(&g, 0, sizeof(g));
    for (int i = 0; i < n_spatial_dims; i++) g.sdims[i] = spatial_dims[i];
    g.spatial_std_d = spatial_std;
    g.feature_std_d = feature_std;
    positions_kernel_f64<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        reference, positions, n, n_reference_channels, n_spatial_dims, g);
    PL_CUDA(cudaGetLastError());
    return PL_OK;
}

static int filter_common_f64(const Geom& g, double* output, const double* input, const double* positions,
                             const double* reference, int pd, int vd, int reverse, void* workspace,
                             size_t workspace_bytes, int64_t max_entries, cudaStream_t st) {
    Layout L;
    int rc = make_layout(L, g, pd, vd, max_entries, 8);
    if (rc != PL_OK) return rc;
    if (workspace_bytes < L.total) return PL_WORKSPACE_TOO_SMALL;
#define CALL(P) run_filter_f64<P>(g, output, input, positions, reference, vd, reverse, workspace, L, st)
    PL_DISPATCH_PD(pd, CALL)
#undef CALL
}

int pl_filter_f64(double* output, const double* input, const double* positions, int batch, int n, int pd,
                  int vd, int reverse, void* workspace, size_t workspace_bytes, int64_t max_entries,
                  void* stream) {
    WatchScope this_call;
    if (batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || !positions || !workspace) return PL_INVALID_ARGUMENT;
    Geom g;
    int one = n;
    int rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    if (rc != PL_OK) return rc;
    set_geom_f64(g, pd, 1.0, 1.0);
    return filter_common_f64(g, output, input, positions, nullptr, pd, vd, reverse, workspace, workspace_bytes,
                             max_entries, (cudaStream_t)stream);
}

int pl_lattice_filter_f64(double* output, const double* input, const double* reference, int batch,
                          int n_spatial_dims, const int* spatial_dims, int n_input_channels,
                          int n_reference_channels, int bilateral, double theta_alpha, double theta_beta,
                          double theta_gamma, int reverse, void* workspace, size_t workspace_bytes,
                          int64_t max_entries, void* stream) {
    WatchScope this_call;
    if (n_input_channels < 1) return PL_INVALID_ARGUMENT;
    Geom g;
    int pd = 0, n = 0;
    int rc = op_geom(g, batch, n_spatial_dims, spatial_dims, n_reference_channels, bilateral, (float)theta_alpha,
                     (float)theta_beta, (float)theta_gamma, &pd, &n);
    if (rc != PL_OK) return rc;
    set_geom_f64(g, pd, bilateral ? theta_alpha : theta_gamma, bilateral ? theta_beta : -1.0);
    const int vd = n_input_channels + 1;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    if (!output || !input || !workspace || (g.R > 0 && !reference)) return PL_INVALID_ARGUMENT;
    return filter_common_f64(g, output, input, nullptr, reference, pd, vd, reverse, workspace, workspace_bytes,
                             max_entries, (cudaStream_t)stream);
}

int pl_export_lattice_f64(const void* workspace, const double* positions, const double* reference, int batch,
                          int n, int pd, int vd, int n_spatial_dims, const int* spatial_dims,
                          int n_reference_channels, double spatial_std, double feature_std, int64_t max_entries,
                          int64_t max_vertices, int16_t* vertex_keys, int32_t* vertex_item,
                          int32_t* pixel_vertex, double* pixel_weight, void* stream) {
    if (!workspace || batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    Geom g;
    int rc;
    if (positions) {
        int one = n;
        rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    } else {
        if (n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || !spatial_dims ||
            n_spatial_dims + n_reference_channels != pd || (n_reference_channels > 0 && !reference))
            return PL_INVALID_ARGUMENT;
        rc = make_geom(g, batch, n, pd, n_spatial_dims, spatial_dims, n_reference_channels, (float)spatial_std,
                       (float)feature_std, false);
    }
    if (rc != PL_OK) return rc;
    set_geom_f64(g, pd, spatial_std, feature_std);
    Layout L;
    rc = make_layout(L, g, pd, vd, max_entries, 8);
    if (rc != PL_OK) return rc;
#define CALL(P) run_export<P, double, Cfg<P>::KW>(g, positions, reference, workspace, L, (long long)max_vertices, vertex_keys, \
                                      vertex_item, pixel_vertex, pixel_weight, (cudaStream_t)stream)
    PL_DISPATCH_PD(pd, CALL)
#undef CALL
}

int pl_crf_step_f32(float* q_out, const float* q, const float* unaries, float bilateral_weight, float spatial_weight,
                    int n_labels, int batch, int n_spatial_dims, const int* spatial_dims, int n_reference_channels,
                    void* bilateral_workspace, size_t bilateral_bytes, int64_t bilateral_entries, void* spatial_workspace,
                    size_t spatial_bytes, int64_t spatial_entries, void* stream) {
    if (n_labels < 1 || batch < 0 || batch > 65535 || n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || !spatial_dims ||
        n_reference_channels < 0)
        return PL_INVALID_ARGUMENT;
    if (n_spatial_dims != 2 || n_reference_channels != 3 || n_labels < 4 || n_labels > 31) return PL_UNSUPPORTED_DIMS;
    const int pda = n_spatial_dims + n_reference_channels, pds = n_spatial_dims, vd = n_labels + 1;
    long long n = 1;
    for (int i = 0; i < n_spatial_dims; i++) {
        if (spatial_dims[i] < 0) return PL_INVALID_ARGUMENT;
        n *= spatial_dims[i];
        if (n > 0x7FFFFFFFll) return PL_INVALID_ARGUMENT;
    }
    if (batch == 0 || n == 0) return PL_OK;
    if (!q_out || !q || !unaries || !bilateral_workspace || !spatial_workspace) return PL_INVALID_ARGUMENT;
    Geom g;
    PL_TRY(make_geom(g, batch, (int)n, pda, n_spatial_dims, spatial_dims, n_reference_channels, 1.f, 1.f, false));
    const dim3 grid = tile_grid(g);
    if (g.grid3 ? grid.z > 32767u : grid.x > 0x3FFFFFFFu) return PL_UNSUPPORTED_DIMS;   // twice as many in one launch
    Layout LA, LS;
    PL_TRY(make_layout(LA, g, pda, vd, bilateral_entries));
    PL_TRY(make_layout(LS, g, pds, vd, spatial_entries));
    if (bilateral_bytes < LA.total || spatial_bytes < LS.total) return PL_WORKSPACE_TOO_SMALL;
    return run_crf_step<5, 2>(g, q_out, q, unaries, bilateral_weight, spatial_weight, n_labels, bilateral_workspace, LA,
                              spatial_workspace, LS, (cudaStream_t)stream);
}

int pl_crf_update_f32(float* q_out, const float* unaries, const float* q_bilateral, const float* q_spatial,
                      const float* compatibility, float bilateral_weight, float spatial_weight,
                      int64_t n_points, int n_labels, void* stream) {
    if (n_points < 0 || n_labels < 1) return PL_INVALID_ARGUMENT;
    if (n_labels > 128) return PL_UNSUPPORTED_DIMS;
    if (n_points == 0) return PL_OK;
    if (!q_out || !unaries || !q_bilateral || !q_spatial) return PL_INVALID_ARGUMENT;
    return launch_crf_update(q_out, unaries, q_bilateral, q_spatial, compatibility, bilateral_weight, spatial_weight, n_points,
                             n_labels, (cudaStream_t)stream);
}

int pl_crf_start_f32(float* q_out, const float* unaries, int64_t n_points, int n_labels, void* stream) {
    if (n_points < 0 || n_labels < 1) return PL_INVALID_ARGUMENT;
    if (n_labels > 128) return PL_UNSUPPORTED_DIMS;
    if (n_points == 0) return PL_OK;
    if (!q_out || !unaries) return PL_INVALID_ARGUMENT;
    return launch_crf_update(q_out, unaries, nullptr, nullptr, nullptr, 0.f, 0.f, n_points, n_labels, (cudaStream_t)stream);
}

unsigned long long pl_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int pl_direct_index_min_entries(int batch, int n_spatial_dims, const int* spatial_dims, float theta_gamma,
                                int64_t* min_entries) {
    if (!min_entries || !spatial_dims || batch < 0 || n_spatial_dims < 1) return PL_INVALID_ARGUMENT;
    *min_entries = 0;
    if (n_spatial_dims > MAX_SDIMS || !pd_supported(n_spatial_dims) || batch == 0) return PL_OK;
    float scale[MAX_PD];
    scale_factors(n_spatial_dims, scale);
    Direct d;
    if (!direct_bounds(d, n_spatial_dims, spatial_dims, theta_gamma, scale, batch, ~0ull)) return PL_OK;
    // the index uses the hash table's region as 32-bit slots: 2 * table slots, table slots >= 2 * max_entries
    *min_entries = (int64_t)((d.slots + 3) / 4);
    return PL_OK;
}

int pl_debug_direct_index(int enable) {
    const int was = g_direct_index_enabled;
    g_direct_index_enabled = enable ? 1 : 0;
    return was;
}

int pl_profile_next_call(void** stage_events) {
    g_stage_events = reinterpret_cast<cudaEvent_t*>(stage_events);
    return PL_OK;
}

int pl_watch_next_call(void* stream) {
    Watcher& w = g_watcher;
    w.armed = w.launched = false;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    PL_CUDA(cudaStreamIsCapturing((cudaStream_t)stream, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        snprintf(g_cuda_error, sizeof(g_cuda_error), "pl_watch_next_call: the stream is being captured");
        return PL_CUDA_ERROR;
    }
    if (!w.line) {
        const int rc = take_watch_line(&w.line);
        if (rc != PL_OK) return rc;
    }
    const int late = take_late_failure(w.line);
    if (late != PL_OK) {
        snprintf(g_cuda_error, sizeof(g_cuda_error),
                 "pl_watch_next_call: an earlier watched call failed after its report, its output holds NaN");
        return late;
    }
    w.line->seq = (w.line->seq + 1) & WATCH_SEQ_MASK;
    if (w.line->seq == 0) w.line->seq = 1;
    w.armed = true;
    return PL_OK;
}

int pl_watched_calls_status(int* device_status) {
    if (!device_status) return PL_INVALID_ARGUMENT;
    *device_status = PL_OK;
    std::lock_guard<std::mutex> lock(g_watch_mutex);
    for (WatchLine* page : watch_pages())
        for (int i = 0; i < 64; i++) {
            const int late = take_late_failure(page + i);
            if (late != PL_OK) *device_status = late;
        }
    return PL_OK;
}

int pl_cancel_watch(void) {
    g_watcher.armed = g_watcher.launched = false;
    return PL_OK;
}

// The report of a call whose stream is idle comes within some tens of microseconds: polled without a pause.  Where
// it takes longer (earlier work in the stream), or the process has asked for waits that block, the thread sleeps
// between polls and leaves its core to others; the sleep, 50 to 100 us with the system's timer slack, is then small
// beside the wait and beside what the device still has to do after the report.
constexpr auto WATCH_SPIN = std::chrono::microseconds(1000), WATCH_NAP = std::chrono::microseconds(20);

int pl_await_watched_call(int64_t* num_entries, int* device_status, void* stream) {
    Watcher& w = g_watcher;
    w.armed = false;
    if (!num_entries || !device_status || !w.launched) return PL_INVALID_ARGUMENT;
    w.launched = false;
    volatile u64* word = &w.line->words[0];
    const auto start = std::chrono::steady_clock::now();
    bool drained = false, nap = false;
    for (unsigned spin = 1;; spin++) {
        const u64 v = *word;
        if ((u32)(v >> 40) == w.line->seq) {
            *num_entries = (int64_t)(u32)v;
            *device_status = code_of((v >> 32) & 0xFFu);
            return PL_OK;
        }
        if (drained) {
            snprintf(g_cuda_error, sizeof(g_cuda_error), "pl_await_watched_call: the call ended without a report");
            return PL_CUDA_ERROR;
        }
        // now and then: has the stream failed, or run empty (then the report is there, or never comes)?
        if (nap || (spin & 0xFFFu) == 0) {
            const cudaError_t e = cudaStreamQuery((cudaStream_t)stream);
            if (e != cudaSuccess && e != cudaErrorNotReady) return cuda_fail(e, "pl_await_watched_call");
            drained = e == cudaSuccess;
            unsigned flags = 0;
            if (!nap && cudaGetDeviceFlags(&flags) == cudaSuccess)
                nap = (flags & cudaDeviceScheduleMask) == cudaDeviceScheduleBlockingSync ||
                      std::chrono::steady_clock::now() - start > WATCH_SPIN;
            if (nap && !drained) std::this_thread::sleep_for(WATCH_NAP);
        }
#if defined(__x86_64__) && !defined(__CUDA_ARCH__)
        if (!nap) __builtin_ia32_pause();
#endif
    }
}

int pl_lattice_stats(const void* workspace, pl_stats* stats, void* stream) {
    if (!stats) return PL_INVALID_ARGUMENT;
    if (!workspace) {   // the built-in scratch of pl_lattice_filter_f32_noalloc on the current device
        void* scratch = nullptr;
        const int rc = static_scratch_of_current_device(&scratch);
        if (rc != PL_OK) return rc;
        workspace = scratch;
    }
    Header h;
    PL_CUDA(cudaMemcpyAsync(&h, workspace, sizeof(Header), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    PL_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    const u32 items = h.items > 1 ? h.items : 1;   // (see one_for_all)
    stats->num_vertices = (int64_t)h.num_vertices * items;
    stats->num_entries = (int64_t)h.num_entries * items;
    stats->table_slots = (int64_t)1 << h.table_log2;
    stats->device_status = PL_OK;
    for (int code = PL_INVALID_ARGUMENT; code <= PL_INTERNAL_ERROR; code++)
        if (h.status & (1u << code)) stats->device_status = code;
    stats->direct_index = (int32_t)h.direct;
    stats->max_entries = (int64_t)h.capacity;
    return PL_OK;
}

int pl_export_lattice(const void* workspace, const float* positions, const float* reference,
                      int batch, int n, int pd, int vd, int n_spatial_dims, const int* spatial_dims,
                      int n_reference_channels, float spatial_std, float feature_std,
                      int64_t max_entries, int64_t max_vertices, int16_t* vertex_keys,
                      int32_t* vertex_item, int32_t* pixel_vertex, float* pixel_weight,
                      void* stream) {
    if (!workspace || batch < 0 || n < 0 || batch > 65535) return PL_INVALID_ARGUMENT;
    if (!pl_supported(pd, vd)) return PL_UNSUPPORTED_DIMS;
    if (batch == 0 || n == 0) return PL_OK;
    Geom g;
    int rc;
    if (positions) {
        int one = n;
        rc = make_geom(g, batch, n, pd, 1, &one, pd - 1, 1.f, 1.f, true);
    } else {
        if (n_spatial_dims < 1 || n_spatial_dims > MAX_SDIMS || !spatial_dims ||
            n_spatial_dims + n_reference_channels != pd || (n_reference_channels > 0 && !reference))
            return PL_INVALID_ARGUMENT;
        rc = make_geom(g, batch, n, pd, n_spatial_dims, spatial_dims, n_reference_channels,
                       spatial_std, feature_std, false);
    }
    if (rc != PL_OK) return rc;
    Layout L;
    rc = make_layout(L, g, pd, vd, max_entries);
    if (rc != PL_OK) return rc;
#define CALL(P) (batch_of_one(g) ? run_export<P, float, Cfg<P>::KW_ALONE> : run_export<P, float, Cfg<P>::KW>)(g, positions, reference, workspace, L, (long long)max_vertices, vertex_keys, \
                                     vertex_item, pixel_vertex, pixel_weight, (cudaStream_t)stream)
    PL_DISPATCH_PD(pd, CALL)
#undef CALL
}

}  // extern "C"
