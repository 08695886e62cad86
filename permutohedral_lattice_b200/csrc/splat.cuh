// Splat stage: per-tile sort of the splats by entry and segmented reduction into the vertex rows
// (a thread per window of narrow rows, a group of lanes per window of wider ones; float and fixed-point sums); tiles with
// few entries by columns of points, unsorted.
#pragma once
#include <type_traits>
#include "common.cuh"

namespace pl {

// ---------------------------------------------------------------------------------------------
// splat_tiles: V[vertex] += sum over the tile's splats of weight * [input channels, 1].
// The splats of a tile are counting-sorted by entry in shared memory, then every entry's run is
// summed in registers, reading the tile's input rows from shared memory, and leaves the CTA as one
// vector reduction per 16 bytes.  No floating-point atomics in shared memory.
//
// Rows of one float4 (splat_tiles_fast): one THREAD sums a window of PD+1 sorted splats with the whole
// row in registers; the input block arrives by bulk asynchronous copies when its rows are 16-byte aligned.
// Wider rows (splat_tiles_rows): a group of lanes per window, see there.
// ---------------------------------------------------------------------------------------------
// A sorted splat: point | entry << 16, and its weight.
__device__ __forceinline__ uint2 splat_record(unsigned key, float w) { return make_uint2(key, __float_as_uint(w)); }
__device__ __forceinline__ uint4 splat_record(unsigned key, double w) {
    return make_uint4(key, 0u, (unsigned)__double2loint(w), (unsigned)__double2hiint(w));
}

template <int PD>
struct SplatCommon {
    static constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, NW = TP / 32;
    // Words of the sorted list with one spare word a window of PD + 1 splats.
    static constexpr int SORTED = SPLATS + TP;

    // Sorted position pos is stored at slot(pos).  Splats of one entry, written together by neighbouring lanes, land in
    // neighbouring words either way.
    // WL = Cfg<PD>::WL (a group of lanes per window, 16 bytes a load): stretches of WL splats, two spare words after each,
    // see there.
    // WL = PD + 1 (a thread per window, 8 bytes a load): one spare word a window, so that lanes in step read words PD + 2
    // apart: an odd distance, and no two on one bank, where PD is odd (5 above all).
    template <int WL>
    __device__ static __forceinline__ int slot(int pos) {
        if constexpr (WL == Cfg<PD>::WL)
            return Cfg<PD>::srec_slot(pos);
        else
            return pos + pos / WL;
    }

    // Counting sort of the tile's splats by entry.  On return (after the trailing barrier) entry e's
    // splats are the sorted positions from cur_s[e] on, each stored as
    // (point | entry << 16, weight) (splat_record).
    // cur_s must be zero for e < nloc on entry.  One shared-memory atomic per splat: the value it
    // returns is the splat's offset inside its entry's run, so no second atomic pass is needed once the
    // run starts are known.  (Grouping equal entries of a warp with a match instruction first measured
    // slower than letting the atomics collide.)
    template <int WL, typename Rec, typename W>
    __device__ static __forceinline__ void sort_splats(bool valid, const int* l, const W* w, int nloc,
                                                       Rec* sorted_s, int* cur_s, int* wsum_s) {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        int off[PD + 1];
#pragma unroll
        for (int r = 0; r <= PD; r++) off[r] = valid ? atomicAdd(&cur_s[l[r]], 1) : 0;
        __syncthreads();
        int local[PD + 1];
        int sum = 0;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int i = tid * (PD + 1) + r;
            local[r] = sum;
            sum += (i < nloc) ? cur_s[i] : 0;
        }
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += t;
        }
        if (lane == 31) wsum_s[warp] = incl;
        __syncthreads();
        int before = 0;   // entries' splats counted by the warps below this one (NW broadcast reads, no second barrier)
#pragma unroll
        for (int q = 0; q < NW; q++) before += (q < warp) ? wsum_s[q] : 0;
        const int excl = incl - sum + before;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int i = tid * (PD + 1) + r;
            if (i < nloc) cur_s[i] = excl + local[r];
        }
        __syncthreads();
        if (valid) {
#pragma unroll
            for (int r = 0; r <= PD; r++) {
                const int pos = cur_s[l[r]] + off[r];
                sorted_s[slot<WL>(pos)] = splat_record((unsigned)tid | ((unsigned)l[r] << 16), w[r]);
            }
        }
        __syncthreads();
    }
};

// A splat kernel that expects sorted splats met a lattice without them (pl_lattice_apply_f32 on a workspace
// that no pl_lattice_build*_f32 prepared): the call fails, its output is poisoned by the slice stage.
__device__ __forceinline__ bool lattice_is_sorted(Header* hdr) {
    if (hdr->sorted) return true;
    if (threadIdx.x == 0) atomicOr(&hdr->status, 1u << PL_INVALID_ARGUMENT);
    return false;
}

// The tile's splats as build_tiles sorted them (entry order; (point | entry << 16, weight bits) each),
// copied into the windowed shared-memory list.  The caller's next barrier publishes them.
template <int PD, int WL>
__device__ __forceinline__ void load_sorted_splats(const uint2* __restrict__ srec_tile, int total, uint2* sorted_s) {
    constexpr int TP = Cfg<PD>::TP;
    uint2 v[PD + 1];
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        const int pos = r * TP + (int)threadIdx.x;
        v[r] = (pos < total) ? srec_tile[Cfg<PD>::srec_slot(pos)] : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        const int pos = r * TP + (int)threadIdx.x;
        if (pos < total) sorted_s[SplatCommon<PD>::template slot<WL>(pos)] = v[r];
    }
}

// PRE: the lattice was built for reuse and holds every tile's splats already sorted (build_tiles with
// SORTED = true); the kernel copies that list instead of sorting the tile's records.
template <int PD, int VD, bool PRE>
struct SplatFast {
    static constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, C = VD - 1;
    static constexpr size_t IN_BYTES = ((sizeof(float) * TP * C + 15) / 16) * 16;
    static constexpr int SORTED = SplatCommon<PD>::SORTED;
    static constexpr size_t BYTES = IN_BYTES + sizeof(uint2) * SORTED + (PRE ? 1 : 2) * sizeof(int) * SPLATS + sizeof(int) * TP;
};

// Adds a row held in registers to vertex row `vrow` (VP floats, 16-byte aligned).
template <int VP>
__device__ __forceinline__ void flush_row(float* vrow, float* acc) {
#pragma unroll
    for (int q = 0; q < VP / 4; q++)
        red_add_v4(vrow + 4 * q, make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]));
#pragma unroll
    for (int j = 0; j < VP; j++) acc[j] = 0.f;
}

// A tile with few entries for its splats (a volume, a smooth guide): points next to one another mostly share their
// vertices, so that walking down a piece of a column of points meets about as few runs as the sorted list cut into windows
// does, and needs no sort.  One thread a piece and remainder; nothing goes through shared memory: a point's row is read
// PD + 1 times, from L1 after the first, neighbouring threads on neighbouring points.  Sixteen points are cut into as many
// pieces as give every thread one (5, 4 and 3 with pd 2, 3 and 4), or two where many tiles share a vertex.
// Bound by the latency of its loads (most stalls are for them; its reductions are none, L2 is at 34 %).  Two volumes of
// 111x128x120 points, 20 splats an entry: sorted 106 us (LSU pipe at 82 %), in columns of eight points, which left 3 of 8 warps
// without work, 87, so 83.  us a call, eight points / so: 16 x 512x512 x 1 without a guide 208 / 186, x 3 198 / 189; 96x128x128 x
// 1 without a guide, forward + backward, 207 / 200.  (The figures below are those of eight points.)  At pd 4 the records of
// one and two channels are loaded evict-first, which leaves L1 to the points' rows.  us a call, plain / so, volumes of 0.5 to 8 M points and
// images of 1 to 4 M: one channel 64x80x96 64.7 / 64.8, two of them 86.1 / 86.8, two of 111x128x120 262.6 / 258.8 (theta 10: 255 / 247),
// 200x200x200 552 / 550, images 105.3
// / 105.4 to 308 / 308; two channels 54.6 / 54.7, 87 / 87, 263 / 260 (253 / 247), 555 / 555.5, images 94.4 / 94.6 to 315.2 / 315.5.  Not with
// three, 56 / 56.5, 88.6 /
// 89.7, 268 / 269 (259 / 257), 568 / 577, images 96 / 97 to 324 / 326, nor at pd 3: 8 volumes of 64x64x64 without a guide 75 / 74, 83 / 84 and 83
// / 83.
// Where (us a splat, columns / sorted): rows of more than one float4 from 2 pd splats an entry on (8 x 512x512, pd 2,
// 21 channels, 4.8 splats 95 / 110, 14.7 splats 76 / 98); narrow ones as NarrowColumns says.  pd 5, us a call: 8
// splats an entry 201 / 197, 36 splats 158 / 138: up to pd 4.  Tiles of points in one dimension, which are all there are with pd 1, have no columns.
constexpr int COLUMN = 8;   // points of a column, wide rows
template <int PD>
__device__ __forceinline__ bool in_columns(const Geom& g, int entries, int least) {   // least: splats an entry
    return g.TX <= 16 && least * entries <= Cfg<PD>::SPLATS;
}
// Rows of one float4, VD - 1 channels.  Sorted tiles want the 32 registers of eight CTAs an SM (pd 2 and 3; also pd 4
// in a kept lattice), columns of four points ahead want 40: with those, and 24 to 56 bytes spilled, sorted tiles took
// 10 to 17 % longer (pd 2, 1 channel, 3.5 splats an entry 41 -> 48 us; 36 -> 42 in a kept lattice).  Two points ahead
// fit 32 registers (up to 8 bytes spilled).  pd 4 sorts with 40 registers anyway.  With two channels, four points
// ahead gain more in columns than they cost sorted tiles (pd 2, 14.7 splats an entry 37 us, two ahead 41, sorted 45;
// 3.5 splats, sorted with six CTAs 49, with eight 43; pd 3, 12.6 splats 43, two ahead 45, sorted 50; kept lattices
// only at pd 2).  From how many splats an entry on, us a splat, columns / sorted: pd 2, 1 channel, 8 splats 47 / 39,
// 14.7 splats 43 / 43, 38 splats 39 / 49; 2 channels, 8 splats 42 / 43; 3 channels, 14.7 splats 44 / 47.  pd 3, 1 and
// 3 channels, 6.6 splats 1.06 to 1.12 of the sort's time, 12.6 splats 0.92 to 0.96; 2 channels, 6.6 splats 1.00, 8.9
// splats 0.93.  pd 4, 9.8 splats 0.88 to 1.04, 20 splats 0.82 to 0.96.  Kept lattices, sorted already: pd 2 and 3
// with 2 channels from 8 and 10 splats on, with 1 and 3 channels 1.03 to 1.10 at 15 splats, 0.91 to 1.09 beyond 26;
// pd 4 never faster.
template <int PD, int VD, bool PRE>
struct NarrowColumns {
    static constexpr bool EVER = PD >= 2 && PD <= (PRE ? 3 : 4);
    static constexpr int AHEAD = PD == 4 ? 3 : VD == 3 && (PD == 2 || !PRE) ? 4 : 2;
    static constexpr int CTAS = !EVER ? 0 : AHEAD >= 3 ? 6 : 8;
    // Where a vertex is shared by more tiles (entries a vertex), what counts is how often they add to it: pieces of eight points then.  us
    // a call, pieces of 3 to 5 points / of eight: pd 2, 3 tiles a vertex 98.7 / 101.3, 4.5 104.7 / 101.3, 21 165 / 119, 76 381 / 199; pd 3, 6.8 79.0 / 80.0,
    // 7 to 8 195 / 204 and 35.3 / 33.7, 26 95.6 / 86.2, 111 214 / 145; pd 4, 12.5 223 / 229, 18.8 75 / 72, 78 366 / 311.
    static constexpr u32 SHARED = PD == 2 ? 4 : PD == 3 ? 10 : 16;
    static constexpr int LEAST = AHEAD >= 3 ? 8 : !PRE ? (PD == 2 ? 12 : 10) : VD == 3 ? 10 : 24;
};
// Few entries are not enough where a noisy guide sends neighbouring points to one and another of them: a column then
// meets a run nearly every point, and all tiles add to few vertices.  So tiles that have more entries than one under
// a flat guide would (Geom::calm_entries) are sampled for changes of entry from one row to the next.  A smooth guide,
// or none, gives 3 to 7 changes an entry, whatever its scale, noise 9 to 24.  Columns or sorted, us a splat: 4 x
// 512x512 guided by one channel, 2 channels, 12 changes 27 / 35, 15 changes 41 / 48, 18 changes 73 / 72, 23 changes
// 74 / 51; guided by two channels, 7 changes 31 / 39, 9 and 13 changes 51 / 35 and 42 / 39; two noisy volumes of
// 96x128x128, 5 changes 84 / 96, 13 changes 275 / 190.  Rows of 21 channels: 12 changes 53 / 61, 15 changes 64 / 62,
// 18 changes 94 / 62, 23 changes 109 / 61, and volumes with 4 changes but fewer than 12 entries a tile 148 / 119.
// With pd 2 there is no guide.  Every warp looks at the same 64 pairs of points, so that all agree without a barrier;
// it costs those tiles 4 to 7 %.  (All tiles sampled cost the splat of smooth volumes 7 %; all points of every second
// row, counted over the CTA, 4 to 20 %; counted by build_tiles, that 3 to 6 %.)
template <int PD>
struct ColumnsSample {
    static constexpr bool TAKEN = PD == 3 || PD == 4;
    static constexpr int NARROW = PD == 4 ? 8 : 16, WIDE = 12;   // changes an entry, at most
    __device__ static __forceinline__ bool smooth(const Geom& g, const TilePos& tpos, const Header* hdr,
                                                  const u16* __restrict__ rec, int entries, int most) {   // TX <= 16
        if (!TAKEN || entries <= (int)hdr->calm_entries) return true;
        const u16* rec_tile = rec + (size_t)tpos.tile * Cfg<PD>::SPLATS + (threadIdx.x & 31);
        u32 e[4];   // of 32 points each, two rows of 16 or more shorter ones, in four remainders
#pragma unroll
        for (int k = 0; k < 4; k++) e[k] = rec_tile[(k % (PD + 1)) * Cfg<PD>::TP + 64 * k];
        int changes = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int row = (64 * k + ((int)threadIdx.x & 31)) >> g.tx_log2;
            const u32 above = __shfl_up_sync(0xFFFFFFFFu, e[k], g.TX);
            changes += __popc(__ballot_sync(0xFFFFFFFFu, (row & 1) && tpos.ty * g.TY + row < g.H && e[k] != above));
        }
        return 4 * (PD + 1) * changes <= most * entries;
    }
};
template <int PD, int VD, int AHEAD>
__device__ __forceinline__ void splat_columns(const Geom& g, const TilePos& tpos, int base,
                                              const float* __restrict__ input, const u16* __restrict__ rec_tile,
                                              const float* __restrict__ recw_tile,
                                              const u32* __restrict__ list_ref, float* __restrict__ v0, bool halves) {
    constexpr int TP = Cfg<PD>::TP, C = VD - 1, VP = (VD + 3) & ~3;
    constexpr bool ONCE = PD == 4 && VD <= 3;   // (see above)
    constexpr int PIECES = TP / (16 * (PD + 1));   // of 16 points of a column, or two; a tile has TX columns of 256 / TX points
    const int tid = threadIdx.x, r = halves ? tid / 32 : tid / (16 * PIECES), c = halves ? tid % 32 : tid % (16 * PIECES);
    const int lx = c & (g.TX - 1), s = c >> g.tx_log2, k = halves ? s % 2 : s % PIECES;
    const int from = halves ? 8 * k : 16 * k / PIECES, to = halves ? from + 8 : 16 * (k + 1) / PIECES;
    const int ly = (halves ? s / 2 : s / PIECES) * 16 + from;
    const int x = tpos.tx * g.TX + lx, y = tpos.ty * g.TY + ly;
    const int rows = r <= PD && x < g.W ? min(to - from, g.H - y) : 0;
    if (rows <= 0) return;
    const u16* rp = rec_tile + r * TP + ly * g.TX + lx;
    const float* wp = recw_tile + r * TP + ly * g.TX + lx;
    const float* in = input + ((size_t)tpos.item * g.n + ((size_t)tpos.o * g.H + y) * g.W + x) * C;
    const size_t step = (size_t)g.W * C;
    float acc[VP];
#pragma unroll
    for (int j = 0; j < VP; j++) acc[j] = 0.f;
    u32 cur = list_ref[base + rp[0]];
#pragma unroll 1
    for (int k0 = 0; k0 < rows; k0 += AHEAD) {   // AHEAD points' loads in flight
        u32 v[AHEAD];
        float w[AHEAD], xv[AHEAD][C];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            const bool there = k0 + k < rows;
            v[k] = !there ? 0u : ONCE ? load_record<PD>(rp + (k0 + k) * g.TX) : rp[(k0 + k) * g.TX];
            w[k] = !there ? 0.f : ONCE ? load_record<PD>(wp + (k0 + k) * g.TX) : wp[(k0 + k) * g.TX];
#pragma unroll
            for (int j = 0; j < C; j++) xv[k][j] = there ? __ldg(in + (size_t)(k0 + k) * step + j) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < AHEAD; k++) v[k] = (k0 + k < rows) ? list_ref[base + v[k]] : cur;
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            if (k0 + k < rows) {
                if (v[k] != cur) {
                    flush_row<VP>(v0 + (size_t)cur * VP, acc);
                    cur = v[k];
                }
#pragma unroll
                for (int j = 0; j < C; j++) acc[j] = PL_FMA(w[k], xv[k][j], acc[j]);
                acc[C] = PL_FADD(acc[C], w[k]);
            }
        }
    }
    flush_row<VP>(v0 + (size_t)cur * VP, acc);
}

template <int PD, int VD, bool PRE>
__global__ void __launch_bounds__(Cfg<PD>::TP, NarrowColumns<PD, VD, PRE>::CTAS)
splat_tiles_fast(Geom g, const float* __restrict__ input, Header* hdr, const int2* __restrict__ tile_info,
                 const u16* __restrict__ rec, const float* __restrict__ rec_w, const uint2* __restrict__ srec,
                 const u32* __restrict__ list_ref, float* __restrict__ v0, int bulk_ok) {
    wait_for_previous_kernel();
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, C = VD - 1, VP = (VD + 3) & ~3;
    using SF = SplatFast<PD, VD, PRE>;
    using NC = NarrowColumns<PD, VD, PRE>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* in_s = reinterpret_cast<float*>(smem_raw);                                       // [TP][C]
    uint2* sorted_s = reinterpret_cast<uint2*>(smem_raw + SF::IN_BYTES);                    // [SORTED]
    int* prow_s = reinterpret_cast<int*>(sorted_s + SF::SORTED);                            // [TP]
    u32* vid_s = reinterpret_cast<u32*>(prow_s + TP);                                       // [SPLATS] entry -> vertex
    int* cur_s = reinterpret_cast<int*>(vid_s + SPLATS);                                    // [SPLATS], only without PRE
    __shared__ int wsum_s[32];
    __shared__ __align__(8) u64 bar;
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile;
    const int2 info = tile_info[tile];   // (in flight with the status)
    bool halves = false;
    if constexpr (NC::EVER) halves = hdr->num_entries > NC::SHARED * hdr->num_vertices;
    if (call_failed(hdr)) return;
    if (PRE && !lattice_is_sorted(hdr)) return;
    const int base = info.x + first_entry_of<PD>(g, tpos.item), nloc = info.y;
    using CS = ColumnsSample<PD>;
    if constexpr (NC::EVER) {
        if (in_columns<PD>(g, nloc, NC::LEAST) && CS::smooth(g, tpos, hdr, rec, nloc, CS::NARROW)) {
            splat_columns<PD, VD, NC::AHEAD>(g, tpos, base, input, rec + (size_t)tile * SPLATS, rec_w + (size_t)tile * SPLATS,
                                  list_ref, v0, halves);
            return;
        }
    }

    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    for (int i = tid; i < nloc; i += TP) {
        if constexpr (!PRE) cur_s[i] = 0;
        vid_s[i] = list_ref[base + i];
    }
    if (bulk_ok && tid == 0) mbar_init(&bar, 1);
    const int nvalid = __syncthreads_count(valid);

    // stage the tile's input rows in shared memory, [point][channel] without padding: one bulk copy
    // per tile row, each issued by its own thread; thread 0 announces the byte total (nvalid points)
    if (bulk_ok) {
        if (tid == 0) mbar_expect_tx(&bar, (unsigned)nvalid * C * 4u);
        if (tid < g.TY) {
            int first, count;
            if (tile_row(g, tpos, tid, first, count))
                bulk_load(in_s + (size_t)tid * g.TX * C, input + (size_t)first * C, (unsigned)count * C * 4u, &bar);
        }
    } else {
        for (int k = tid; k < TP * C; k += TP) {
            const int p = k / C, j = k - p * C;
            const int row = prow_s[p];
            if (row >= 0) cp_async4(in_s + k, input + (size_t)row * C + j);
        }
    }

    const int total = nvalid * (PD + 1);
    if constexpr (PRE) {
        load_sorted_splats<PD, PD + 1>(srec + (size_t)tile * Cfg<PD>::SREC, total, sorted_s);
    } else {
        float w[PD + 1];
        int l[PD + 1];
        const u16* rec_tile = rec + (size_t)tile * SPLATS;
        const float* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            l[r] = valid ? load_record<PD>(rec_tile + r * TP + tid) : 0;
            w[r] = valid ? load_record<PD>(recw_tile + r * TP + tid) : 0.f;
        }
        SplatCommon<PD>::template sort_splats<PD + 1>(valid, l, w, nloc, sorted_s, cur_s, wsum_s);
    }

    if (bulk_ok) {
        // the outcome of the bounded wait is made uniform over the CTA: either every thread goes on or
        // every thread leaves (after one more bounded wait, so that no copy lands in a CTA that is gone)
        if (!__syncthreads_and(mbar_wait(&bar, 0) ? 1 : 0)) {
            if (tid == 0) atomicOr(&hdr->status, 1u << PL_INTERNAL_ERROR);
            mbar_wait(&bar, 0);
            return;
        }
    } else {
        cp_async_wait_all();
        __syncthreads();
    }

    // Every thread sums a window of PD+1 consecutive sorted splats in registers; whenever the entry
    // changes, and at the end of the window, the partial row leaves as vector reductions.
    const int first = tid * (PD + 1);
    if (first >= total) return;
    float acc[VP];
#pragma unroll
    for (int j = 0; j < VP; j++) acc[j] = 0.f;
    // window tid holds sorted positions first .. first + PD in words tid (PD + 2) + i
    const uint2* sp = sorted_s + tid * (PD + 2);
    int cur = (int)(sp[0].x >> 16);
#pragma unroll
    for (int i = 0; i <= PD; i++) {
        if (first + i < total) {
            const uint2 pw = sp[i];
            const int e = (int)(pw.x >> 16);
            if (e != cur) {
                flush_row<VP>(v0 + (size_t)vid_s[cur] * VP, acc);
                cur = e;
            }
            const float wt = __uint_as_float(pw.y);
            const float* x = in_s + (pw.x & 0xFFFFu) * C;
#pragma unroll
            for (int j = 0; j < C; j++) acc[j] = PL_FMA(wt, x[j], acc[j]);
            acc[C] = PL_FADD(acc[C], wt);
        }
    }
    flush_row<VP>(v0 + (size_t)vid_s[cur] * VP, acc);
}

// The deterministic mode's grid (PL_MODE_DETERMINISTIC): every product weight * value is rounded once to a multiple
// of 2^-36 of the next power of two above max(|input|, 1), found by absmax_kernel, and summed as a 64-bit integer, in
// registers and in global memory.  Integer addition is associative, so the sums do not depend on the order in which
// splats, windows or tiles arrive: results are bitwise reproducible.  Finite inputs only.
__device__ __forceinline__ int fixed_exponent(const Header* hdr) {   // 36 - e with 2^e > max(|input|, 1)
    const u32 bits = max(hdr->absmax_bits, __float_as_uint(1.0f));
    return 36 - ((int)((bits >> 23) & 0xFF) - 127 + 1);
}

// What a lane keeps of the running entry: four channels of its sum.
struct FloatSum {
    float4 a;
    __device__ __forceinline__ void start(const Header*) {}
    __device__ __forceinline__ void clear() { a = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void add(float wt, float4 x) {
        const float2 w2 = make_float2(wt, wt);
        const float2 lo = fma2(w2, make_float2(x.x, x.y), make_float2(a.x, a.y));
        const float2 hi = fma2(w2, make_float2(x.z, x.w), make_float2(a.z, a.w));
        a = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    __device__ __forceinline__ void flush(float* row) const { red_add_v4(row, a); }
};
// The same on the fixed-point grid.  A product scaled to the grid, t with |t| <= 2^36 and a little, is an integer
// number of 2^15 (added to 1.5 * 2^38, whose last place that is) plus a rest of at most 2^14, exact in float, whose
// nearest integer the same trick with 1.5 * 2^23 gives: together t rounded to the nearest integer, ties to even.  The
// two halves of a window's sum, of at most 32 (pd + 1) terms, fit 32 bits each.  The weight is scaled, not the product:
// a power of two changes no rounding (a weight that this takes below the normal range loses 2^-22 of a grid step).  Two products an instruction:
// 2 x 512x512 x 21, pd 5, 96 -> 88 us a splat.  (Converting every product to double
// and that to a 64-bit integer took two instructions of a sixteenth of the float rate each.)
struct FixedSum {
    static constexpr float M_HI = 412316860416.f, M_LO = 12582912.f;
    int hi[4], lo[4];
    float scale;
    __device__ __forceinline__ void start(const Header* hdr) {
        scale = __int_as_float((127 + fixed_exponent(hdr)) << 23);
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 4; k++) hi[k] = lo[k] = 0;
    }
    __device__ __forceinline__ void add_two(int k, float2 wt, float2 x) {
        const float2 t = mul2(wt, x);
        const float2 h = add2(t, make_float2(M_HI, M_HI));
        const float2 whole = add2(h, make_float2(-M_HI, -M_HI));
        const float2 l = add2(fma2(whole, make_float2(-1.f, -1.f), t), make_float2(M_LO, M_LO));
        hi[k] += __float_as_int(h.x) - __float_as_int(M_HI);
        hi[k + 1] += __float_as_int(h.y) - __float_as_int(M_HI);
        lo[k] += __float_as_int(l.x) - __float_as_int(M_LO);
        lo[k + 1] += __float_as_int(l.y) - __float_as_int(M_LO);
    }
    __device__ __forceinline__ void add(float wt, float4 x) {
        const float ws = PL_FMUL(wt, scale);
        const float2 w2 = make_float2(ws, ws);
        add_two(0, w2, make_float2(x.x, x.y));
        add_two(2, w2, make_float2(x.z, x.w));
    }
    __device__ __forceinline__ void flush(long long* row) const {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const long long sum = (long long)hi[k] * 32768 + (long long)lo[k];
            if (sum) atomicAdd(reinterpret_cast<u64*>(row + k), (u64)sum);
        }
    }
};

// Rows of more than one float4: a GROUP OF LANES per window, one float4 of the row per lane (LW lanes: the power of
// two that holds the row, a quarter warp for the 22 channels of the dense-CRF workload).  The input block is staged
// with rows padded to VP floats (16-byte aligned), so the lanes of a group read one point's row as consecutive
// float4 words: a 128-bit shared-memory load is served one quarter warp at a time, so with LW = 8 every quarter
// reads its own row without bank conflicts whatever rows the other quarters read.  Lane h keeps
// channels 4h .. 4h+3 of the running sum; the row's channel C is staged as 1 (homogeneous), the padding
// as 0, so the loop has no channel tests.  A flush is one 16-byte vector reduction per lane.
// VD = 0: any width, known at run time only (rows beyond 32 quads are walked once for every 32).
// Sum: float sums into rows of floats, or fixed-point sums into rows of 64-bit integers (V: type of a row's cell).
// PRE: the lattice was built for reuse and holds every tile's splats already sorted, in the windowed form
// (build_tiles with SORTED = true); the list then arrives by one bulk copy, the kernel needs no sort, no
// counters, and fits five CTAs on an SM.
template <int PD, int VD, bool PRE>
struct SplatRows {
    static constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS;
    static constexpr int WL = Cfg<PD>::WL;             // splats between two spare words of the sorted list
    static constexpr int SORTED = Cfg<PD>::SREC;
    static size_t bytes(int vd) {
        return sizeof(float) * TP * (size_t)padded_vd(vd) + sizeof(uint2) * SORTED + (PRE ? 0 : sizeof(int) * SPLATS) +
               sizeof(int) * TP;
    }
};

// Walking columns of points (see splat_columns) for rows of more than one float4, up to pd = WIDE_COLUMNS_PD: a group
// of lanes per column, as below, with the running sums of all PD + 1 remainders, so that a point's row is read once
// instead of PD + 1 times and neither sorted nor spread to padded rows: lanes read single floats, and four
// neighbouring columns with an odd number of channels never meet on a shared-memory bank.  Channel 0 of point (lx,
// ly) lies at ly row_step + lx point_step; `splat_s` holds the vertex and weight of every splat.  8 x 512x512 x 21,
// pd 2: 99 -> 75 us.  (Running sums of four remainders are what the registers of five CTAs an SM hold.) Columns meet
// more runs than the sorted list's windows, each flushed once.  For a float sum that is one reduction of 16 bytes a
// lane, for a fixed-point sum four of 8 bytes.  Fixed-point sums in columns or sorted, us a splat of 8 x 512x512, pd
// 2, by channels, with 5 and with 15 splats an entry: 1-3 channels 99 / 122 and 84 / 112; 4 channels 139 / 146 and
// 101 / 123; 6 channels 168 / 153 and 116 / 128; with 8 splats an entry 10 channels 1.03, 21 channels 1.29 times the
// sort's time.  pd 3: 0.9 to 2.3 times its time, 21 channels 1.5 to 4.  In a kept lattice, whose splats are sorted
// already: 1-3 channels 87 / 101 from 8 splats an entry on, 4-6 channels 1.0 to 1.1 times, beyond pd 2 never faster.
// Hence: pd 2 only, and there rows of one float4, or of two from 4 pd splats an entry on and if the call would have
// to sort.
constexpr int WIDE_COLUMNS_PD = 3, FIXED_COLUMNS_PD = 2;
template <int PD, bool PRE, typename Sum>
struct WideColumns {
    static constexpr bool FIXED = !std::is_same<Sum, FloatSum>::value;
    static constexpr bool EVER = PD >= 2 && PD <= (FIXED ? FIXED_COLUMNS_PD : WIDE_COLUMNS_PD);
    __device__ static __forceinline__ bool take(const Geom& g, int entries, int LR) {
        if (!EVER) return false;
        if (FIXED) return LR <= (PRE ? 1 : 2) && in_columns<PD>(g, LR * entries, 2 * PD);
        if (PD == 3 && entries < 12) return false;
        // (up to 64 floats a row: a column of as many points as lanes fits the tile)
        return LR <= 16 && in_columns<PD>(g, entries, 2 * PD);
    }
};
template <int PD, typename Sum, typename V>
__device__ __forceinline__ void splat_wide_columns(const Geom& g, const TilePos& tpos, const Header* hdr,
                                                   const float* in_s, int point_step, int row_step, const uint2* splat_s,
                                                   V* __restrict__ v0, int C, int VP) {
    constexpr int TP = Cfg<PD>::TP;
    const int LR = VP >> 2;
    const int lw_log2 = LR > 8 ? 4 : LR > 4 ? 3 : LR > 2 ? 2 : 1, LW = 1 << lw_log2;
    const int points = LW > COLUMN ? LW : COLUMN;   // of a column
    const int c = (int)threadIdx.x >> lw_log2, lx = c & (g.TX - 1), ly = (c >> g.tx_log2) * points;
    const int x = tpos.tx * g.TX + lx, y = tpos.ty * g.TY + ly;
    const int count = (c < TP / points && x < g.W) ? min(points, g.H - y) : 0;
    if (count <= 0) return;
    for (int h = (int)threadIdx.x & (LW - 1); h < LR; h += LW) {
        const uint2* sp = splat_s + ly * g.TX + lx;
        const float* in = in_s + ly * row_step + lx * point_step + 4 * h;
        const int left = C - 4 * h;   // channels from here on; then the homogeneous one, then padding
        Sum acc[PD + 1];
        u32 cur[PD + 1];
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            acc[r].start(hdr);
            acc[r].clear();
            cur[r] = sp[r * TP].x;
        }
#pragma unroll 2
        for (int i = 0; i < count; i++, in += row_step, sp += g.TX) {
            float4 q = make_float4(left == 0 ? 1.f : 0.f, left == 1 ? 1.f : 0.f, left == 2 ? 1.f : 0.f, left == 3 ? 1.f : 0.f);
            if (left > 0) q.x = in[0];
            if (left > 1) q.y = in[1];
            if (left > 2) q.z = in[2];
            if (left > 3) q.w = in[3];
#pragma unroll
            for (int r = 0; r <= PD; r++) {
                const uint2 vw = sp[r * TP];
                if (vw.x != cur[r]) {
                    acc[r].flush(v0 + (size_t)cur[r] * VP + 4 * h);
                    acc[r].clear();
                    cur[r] = vw.x;
                }
                acc[r].add(__uint_as_float(vw.y), q);
            }
        }
#pragma unroll
        for (int r = 0; r <= PD; r++) acc[r].flush(v0 + (size_t)cur[r] * VP + 4 * h);
    }
}

template <int PD, int VD, bool PRE, typename Sum, typename V>
__device__ __forceinline__ void splat_rows(const Geom& g, const TilePos& tpos, const float* __restrict__ input, Header* hdr,
                                           const int2* __restrict__ tile_info, const u16* __restrict__ rec,
                                           const float* __restrict__ rec_w, const uint2* __restrict__ srec,
                                           const u32* __restrict__ list_ref, V* __restrict__ v0, int vd, int bulk_ok) {
    // Launched to overlap the tail of the kernel before it (link_neighbours, or zero_rows in an apply): all
    // that the staging and the sort read (the input, the records and tile ranges of build_tiles, whose
    // failures are final by now) is older than that kernel, so they run before the wait; the window loop,
    // which reads the entries' vertices and adds to the zeroed rows, runs after it.
    using SR = SplatRows<PD, VD, PRE>;
    constexpr int TP = SR::TP, SPLATS = SR::SPLATS, WL = SR::WL;
    const int C = (VD ? VD : vd) - 1, VP = padded_vd(VD ? VD : vd), LR = VP >> 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* in_s = reinterpret_cast<float*>(smem_raw);                         // [TP][VP]
    uint2* sorted_s = reinterpret_cast<uint2*>(in_s + TP * VP);               // [SORTED]
    int* prow_s = reinterpret_cast<int*>(sorted_s + SR::SORTED);              // [TP]
    int* cur_s = prow_s + TP;                                                 // [SPLATS], only without PRE
    __shared__ int wsum_s[32];
    __shared__ __align__(8) u64 bar;
    if (call_failed(hdr) || (PRE && !lattice_is_sorted(hdr))) {
        wait_for_previous_kernel();
        return;
    }
    const int tid = threadIdx.x, tile = tpos.tile, lane = tid & 31, warp = tid >> 5;
    const int2 info = tile_info[tile];
    const int base = info.x + first_entry_of<PD>(g, tpos.item), nloc = info.y;
    using CS = ColumnsSample<PD>;
    constexpr bool SAMPLED = CS::TAKEN && WideColumns<PD, PRE, Sum>::EVER;
    bool columns = WideColumns<PD, PRE, Sum>::take(g, nloc, LR);   // (so far; then by the sample)
    auto look_at_sample = [&]() {
        if constexpr (SAMPLED) {
            if (columns) columns = CS::smooth(g, tpos, hdr, rec, nloc, CS::WIDE);
        }
    };
    if constexpr (PRE) look_at_sample();   // which decides what is loaded

    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    // without PRE the splat records are loaded first: they depend on nothing but the tile number, so their
    // latency overlaps that of the tile's entry range above
    float w[PD + 1];
    int l[PD + 1];
    if (!PRE || columns) {
        const u16* rec_tile = rec + (size_t)tile * SPLATS;
        const float* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            l[r] = valid ? load_record<PD>(rec_tile + r * TP + tid) : 0;
            w[r] = valid ? load_record<PD>(recw_tile + r * TP + tid) : 0.f;
        }
    }
    if (!PRE)
        for (int i = tid; i < nloc; i += TP) cur_s[i] = 0;
    if ((PRE || bulk_ok) && tid == 0) mbar_init(&bar, 1);
    const int nvalid = __syncthreads_count(valid);
    const int total = nvalid * (PD + 1);
    // PRE: the tile's sorted splats arrive by one bulk copy, already in the windowed form the loop below reads
    const unsigned rec_bytes = PRE && !columns ? (unsigned)(sizeof(uint2) * SR::SORTED) : 0u;
    if ((PRE || bulk_ok) && tid == 0) {
        mbar_expect_tx(&bar, rec_bytes + (bulk_ok ? (unsigned)nvalid * C * 4u : 0u));
        if (rec_bytes) bulk_load(sorted_s, srec + (size_t)tile * SR::SORTED, rec_bytes, &bar);
    }

    // Staging.  Bulk form: every tile row's block (TX points x C floats, contiguous in memory) lands
    // by one bulk asynchronous copy at the END of the tile row's padded region; after the sort a warp
    // spreads it out in place to the padded rows (all reads of a tile row, then all writes: the
    // landing zone overlaps the rows it feeds).  Otherwise: 4-byte asynchronous copies straight to
    // the padded positions.
    const int land = g.TX * (VP - C);   // floats between the start of a tile row's region and its landing zone
    if (bulk_ok) {
        if (tid < g.TY) {
            int first, count;
            if (tile_row(g, tpos, tid, first, count))
                bulk_load(in_s + (size_t)tid * g.TX * VP + land, input + (size_t)first * C, (unsigned)count * C * 4u,
                          &bar);
        }
    } else {
        in_s[tid * VP + C] = 1.f;   // homogeneous channel, then padding
        for (int j = C + 1; j < VP; j++) in_s[tid * VP + j] = 0.f;
        // element k = tid, tid + TP, ... of the tile's [point][channel] block; (point, channel) advance
        // without a division: TP = DP * C + DJ
        const int DP = TP / C, DJ = TP - DP * C;
        int p = tid / C, j = tid - p * C;
#pragma unroll 3
        for (int it = 0; it < C; it++) {
            const int row = prow_s[p];
            if (row >= 0) cp_async4(in_s + p * VP + j, input + (size_t)row * C + j);
            p += DP;
            j += DJ;
            if (j >= C) {
                j -= C;
                p++;
            }
        }
    }

    if constexpr (!PRE) {
        look_at_sample();   // (from L1 by now, and behind the staging, whose copies it does not hold up)
        if (!columns) SplatCommon<PD>::template sort_splats<WL>(valid, l, w, nloc, sorted_s, cur_s, wsum_s);
    }
    // did this thread see the copies complete within the bounded wait
    const bool arrived = (PRE || bulk_ok) ? mbar_wait(&bar, 0) : true;
    if (bulk_ok && columns) {
        // a column's points are read where they landed
    } else if (bulk_ok) {
        // elements a lane reads before the first of them is written: the whole tile row (TX <= 16) where its size is
        // known, else four at a time (an element moves towards the region's start and the elements after it lie
        // behind its old place, so a trip never overwrites what a later one reads)
        constexpr int MAXE = VD ? (16 * (VD - 1) + 31) / 32 : 4;
        for (int ly = warp; ly < g.TY; ly += TP / 32) {
            // valid points of this tile row: its first point's validity and the row's width
            const int p0 = ly * g.TX;
            const int row0 = prow_s[p0];
            int count = 0;
            if (row0 >= 0) {
                const int x0 = (row0 % g.n) % g.W;
                count = min(g.TX, g.W - x0);
            }
            float* region = in_s + (size_t)p0 * VP;
            const int n = count * C;
            int pp = lane / C, jj = lane - pp * C;   // element e = lane + 32 m is channel jj of point pp
            const int dp = 32 / C, dj = 32 - dp * C;
#pragma unroll 1
            for (int e0 = lane; e0 - lane < n; e0 += 32 * MAXE) {
                float tmp[MAXE];
                int dst[MAXE];
#pragma unroll
                for (int m = 0; m < MAXE; m++) {
                    const int e = e0 + 32 * m;
                    tmp[m] = (e < n) ? region[land + e] : 0.f;
                    dst[m] = (e < n) ? pp * VP + jj : -1;
                    pp += dp;
                    jj += dj;
                    if (jj >= C) {
                        jj -= C;
                        pp++;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int m = 0; m < MAXE; m++)
                    if (dst[m] >= 0) region[dst[m]] = tmp[m];
                if constexpr (VD > 0) break;   // one trip
            }
            if (lane < g.TX) {
                region[lane * VP + C] = 1.f;   // homogeneous channel, then padding
                for (int j = C + 1; j < VP; j++) region[lane * VP + j] = 0.f;
            }
        }
    } else {
        cp_async_wait_all();
    }
    // this barrier also makes the outcome of the bounded wait uniform over the CTA: either every thread
    // goes on or every thread leaves (after one more bounded wait, so that no copy lands in a CTA that
    // is gone)
    if (!__syncthreads_and(arrived ? 1 : 0)) {
        if (tid == 0) atomicOr(&hdr->status, 1u << PL_INTERNAL_ERROR);
        mbar_wait(&bar, 0);
        wait_for_previous_kernel();
        return;
    }
    wait_for_previous_kernel();
    if (call_failed(hdr)) return;   // a failure of the index stage

    if constexpr (WideColumns<PD, PRE, Sum>::EVER) {
        if (columns) {
#pragma unroll
            for (int r = 0; r <= PD; r++)
                sorted_s[r * TP + tid] = make_uint2(valid ? list_ref[base + l[r]] : 0u, __float_as_uint(w[r]));
            __syncthreads();
            splat_wide_columns<PD, Sum>(g, tpos, hdr, in_s + (bulk_ok ? land : 0), bulk_ok ? C : VP, g.TX * VP, sorted_s, v0, C, VP);
            return;
        }
    }

    // (two lanes at least, so that a window starts on an even splat)
    const int lw_log2 = LR > 16 ? 5 : LR > 8 ? 4 : LR > 4 ? 3 : LR > 2 ? 2 : 1;
    const int LW = 1 << lw_log2, wl = LW * (PD + 1);   // lanes of a window, its splats
    const int first = (tid >> lw_log2) * wl, end = min(first + wl, total);
    constexpr bool ONE = VD > 16 && VD <= 32;          // known: a lane has one quad, a window is one stretch
    if (first < end) {
        for (int h = tid & (LW - 1); h < LR; h += LW) {
            const float4* in4 = reinterpret_cast<const float4*>(in_s) + h;
            Sum acc;
            acc.start(hdr);
            acc.clear();
            int cur = (int)(sorted_s[Cfg<PD>::srec_slot(first)].x >> 16);
            u32 vcur = list_ref[base + cur];   // vertex of the running entry, fetched when the run starts
            // a window lies between two spare words of the list, or (LW > 8) is a row of such stretches
            for (int pos = first; pos < end; pos += WL) {
                const uint2* sp = sorted_s + Cfg<PD>::srec_slot(pos);
                const int count = min(WL, end - pos);
                auto one = [&](unsigned key, unsigned weight) {
                    const int e = (int)(key >> 16);
                    if (e != cur) {
                        acc.flush(v0 + (size_t)vcur * VP + 4 * h);
                        acc.clear();
                        cur = e;
                        vcur = list_ref[base + cur];
                    }
                    acc.add(__uint_as_float(weight), in4[(key & 0xFFFFu) * LR]);
                };
                int i = 0;
#pragma unroll 2
                for (; i + 1 < count; i += 2) {   // two splats a load
                    const uint4 pw = *reinterpret_cast<const uint4*>(sp + i);
                    one(pw.x, pw.y);
                    one(pw.z, pw.w);
                }
                if (i < count) one(sp[i].x, sp[i].y);
                if constexpr (ONE) break;
            }
            acc.flush(v0 + (size_t)vcur * VP + 4 * h);
            if constexpr (ONE) break;
        }
    }
}

// Five CTAs per SM (47-48 registers, no spills; with the sort's counters the five CTAs take nearly all of an
// SM's shared memory): 4 % faster than four at 16 items, and 2048 tiles (two items) take three waves, not four.
template <int PD, int VD, bool PRE, typename Sum, typename V>
__global__ void __launch_bounds__(Cfg<PD>::TP, std::is_same<Sum, FloatSum>::value ? 5 : 4)
splat_tiles_rows(Geom g, const float* __restrict__ input, Header* hdr, const int2* __restrict__ tile_info,
                 const u16* __restrict__ rec, const float* __restrict__ rec_w, const uint2* __restrict__ srec,
                 const u32* __restrict__ list_ref, V* __restrict__ v0, int vd, int bulk_ok) {
    splat_rows<PD, VD, PRE, Sum, V>(g, this_tile(g), input, hdr, tile_info, rec, rec_w, srec, list_ref, v0, vd, bulk_ok);
}

// ---------------------------------------------------------------------------------------------
// Deterministic mode: the input's largest magnitude before the splat, the sums as floats after it.
// ---------------------------------------------------------------------------------------------
// One pass over the input, 16 bytes a load and four loads in flight (4-byte loads one by one reached 1.9 TB/s); the up
// to three floats before the first 16-byte boundary and after the last go one by one.  2 x 512x512 x 21, forward +
// backward: 491 -> 466 us.
// It runs beside the kernel after it, whose first part needs nothing of it: the lattice construction, or, in a kept lattice, the
// splat.  Behind the link launch, where it stood alone, 2 x 512x512 x 21, forward + backward, took 414.6 us, so 408.2.
__global__ void __launch_bounds__(256)
absmax_kernel(const float* __restrict__ input, u64 count, Header* hdr) {
    let_next_kernel_start();   // (the input is older than the kernel before this, which has waited: see after_previous_kernel)
    u32 m = 0;
    auto take = [&](float x) { m = max(m, __float_as_uint(fabsf(x))); };
    const u64 lead = min(count, (u64)(((16u - ((u32)(uintptr_t)input & 15u)) & 15u) >> 2));
    const u64 quads = (count - lead) >> 2, tail = lead + 4 * quads, stride = (u64)gridDim.x * blockDim.x;
    const u64 first = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const float4* __restrict__ in4 = reinterpret_cast<const float4*>(input + lead);
    u64 i = first;
    for (; i + 3 * stride < quads; i += 4 * stride) {
        float4 x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = __ldg(in4 + i + k * stride);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            take(x[k].x);
            take(x[k].y);
            take(x[k].z);
            take(x[k].w);
        }
    }
    for (; i < quads; i += stride) {
        const float4 x = __ldg(in4 + i);
        take(x.x);
        take(x.y);
        take(x.z);
        take(x.w);
    }
    if (first < lead) take(input[first]);
    if (first < count - tail) take(input[tail + first]);
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    __shared__ u32 m_s[8];
    if ((threadIdx.x & 31) == 0) m_s[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < 8; k++) m = max(m, m_s[k]);
        wait_for_previous_kernel();   // which zeroes the header's word
        if (m) atomicMax(&hdr->absmax_bits, m);
    }
}

// fixed-point sums -> float rows
__global__ void __launch_bounds__(256)
convert_fixed(const Header* hdr, const long long* __restrict__ v64, float* __restrict__ v0, u32 vp, u64 item_cells) {
    after_previous_kernel();
    v64 += blockIdx.y * item_cells;
    v0 += blockIdx.y * item_cells;
    if (hdr->status != 0) return;
    const double inv = __longlong_as_double((long long)(1023 - fixed_exponent(hdr)) << 52);
    const u64 cells = (u64)hdr->num_vertices * vp;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < cells; i += (u64)gridDim.x * blockDim.x)
        v0[i] = (float)PL_DMUL(__ll2double_rn(v64[i]), inv);
}

// Start of an apply on an already built lattice: value rows (or fixed-point sums) back to zero.  It overlaps the kernel before the call, and the
// kernels after it (absmax_kernel, the splat's staging) read the caller's input before they wait: it must not release them before it has waited.
__global__ void __launch_bounds__(256)
zero_rows(Header* hdr, float* __restrict__ v0, long long* __restrict__ v64, int vp) {
    after_previous_kernel();
    if (hdr->status != 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) hdr->absmax_bits = 0;
    const u64 cells = (u64)hdr->num_vertices * vp;
    const u64 gtid = (u64)blockIdx.x * blockDim.x + threadIdx.x, gsz = (u64)gridDim.x * blockDim.x;
    if (v64) {
        for (u64 e = gtid; e < cells; e += gsz) v64[e] = 0;
    } else {
        for (u64 e = gtid; e < cells; e += gsz) v0[e] = 0.f;
    }
}

}  // namespace pl
