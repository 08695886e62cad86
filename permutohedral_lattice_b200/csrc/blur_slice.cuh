// Blur passes over the vertex rows and the slice stage (interpolate, normalise, write out).
#pragma once
#include <type_traits>
#include "common.cuh"

namespace pl {

// ---------------------------------------------------------------------------------------------
// blur_axis: one [1 2 1]/4 pass along lattice axis `axis` (src/PermutohedralLatticeCPU.h:403-405: the three
// products and their sum in double, one rounding to float; the products are exact, so fusing them into the sums
// changes no bit).  16 bytes of a row per thread (V: float4 or double2).
// Bound by latency at full occupancy: a thread makes few trips of two dependent accesses, the neighbour pair and
// then the rows.  So the pair of the next trip is fetched together with the rows of this one, and a thread goes on
// to its next row without dividing (a 64-bit quotient a trip before).  16 x 512x512 x 21,
// forward + backward (12 passes): 1872 -> 1842 us; 1 M points with 16 features (17 passes): 2048 -> 2014.
// The sums are in double throughout.  What that costs is the conversions, three up and one down a value and sixteen of a warp's a
// cycle and SM, more than half of a pass; so the way up is a move of bits (see moved) where it is faster.  us a call, conversions / moves:
// 16 x 512x512 x 21 1779 / 1766, 375x500 x 21, five steps of a CRF, 442 / 421, 8 x 512x512 x 21 by position alone (pd 2) 428 / 424,
// 1 M points with 16 features 1705 / 1698.  (Floats with the sums' rounding errors added at the end took 1759, 409, 422 and 1691; they are not
// the same bits where the errors' sum fits no float.)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double mix3(double a, double b, double c) {
    return __fma_rn(0.25, c, __fma_rn(0.5, b, PL_DMUL(0.25, a)));
}
__device__ __forceinline__ float mix3(float a, float b, float c) { return (float)mix3((double)a, (double)b, (double)c); }
__device__ __forceinline__ float4 mix_rows(float4 a, float4 b, float4 c) {
    return make_float4(mix3(a.x, b.x, c.x), mix3(a.y, b.y, c.y), mix3(a.z, b.z, c.z), mix3(a.w, b.w, c.w));
}
__device__ __forceinline__ double2 mix_rows(double2 a, double2 b, double2 c) {
    return make_double2(mix3(a.x, b.x, c.x), mix3(a.y, b.y, c.y));
}
// A finite float as a double 2^896 times smaller: its bits as they are, three places down.  The double's exponent counts on
// from 0 as the float's did, and subnormal floats become subnormal doubles.  (Infinities and NaN would become numbers.)
__device__ __forceinline__ double moved(float x) {
    const long long w = (long long)__float_as_int(x) << 29;   // the sign four times over, of which the double has the first
    return __hiloint2double((int)(w >> 32) & 0x8FFFFFFF, (int)w);
}
// The same products as mix3's, exact as there (2^896 / 4 and 2^896 / 2 times the moved numbers): the same sums and bits.
__device__ __forceinline__ float mix3_moved(float a, float b, float c) {
    return (float)__fma_rn(0x1p894, moved(c), __fma_rn(0x1p895, moved(b), PL_DMUL(0x1p894, moved(a))));
}
__device__ __forceinline__ float4 mix_rows_moved(float4 a, float4 b, float4 c) {
    return make_float4(mix3_moved(a.x, b.x, c.x), mix3_moved(a.y, b.y, c.y), mix3_moved(a.z, b.z, c.z),
                       mix3_moved(a.w, b.w, c.w));
}
__device__ __forceinline__ double2 mix_rows_moved(double2 a, double2 b, double2 c) { return mix_rows(a, b, c); }
// z stays zero as long as all numbers given were finite, else it is NaN: which of the two mixes may be taken.
__device__ __forceinline__ void look_for_finite(float2& z, float4 x) {
    const float2 zero = make_float2(0.f, 0.f);
    z = fma2(make_float2(x.z, x.w), zero, fma2(make_float2(x.x, x.y), zero, z));
}
__device__ __forceinline__ void look_for_finite(float2&, double2) {}
__device__ __forceinline__ bool all_finite(float2 z) { return PL_FADD(z.x, z.y) == 0.f; }

// Beyond so many pieces of 16 bytes the rows do not stay in L2, and conversions are as fast as moves or faster: 8 x 512x512 x 21
// of a noisy lattice (20 M pieces) 3768 / 3841 us a call.
constexpr u64 MOVED_ITEMS = 5000000;
// Nor do lines of neighbours that are loaded evict-first stay until the next block wants its part of them, so that beyond it the loop loads them
// plainly: us a call, evict-first / plain, 8 x 512x512 x 21 of a noisy guide, 3.5 M vertices 2577 / 2453, 60 k points x 21 at pd 16, 1 M vertices
// 1056 / 1011.
// Below, evict-first leaves L2 to the rows: 800x1200 x 3 163 / 165, five CRF steps on 375x500 x 21 371 / 378, 200 k points x 7 at pd 16 328 / 341.
// (Two loops: chosen in the loop, it cost up to 4 %.)

template <typename V>
__device__ __forceinline__ void blur_rows(const Header* hdr, const int* __restrict__ nbr_axis, const V* __restrict__ src,
                                          V* __restrict__ dst, u32 vpr /* V per row */, u32 block, u32 blocks, u32 lattices /* of this size */) {
    // Passes after the first overlap the tail of the pass before (see after_previous_kernel).  The vertex count
    // and the neighbour table are older than any blur pass: a thread's first pair of neighbours is fetched
    // before the wait, so that one of the two dependent loads of its first row is off the critical path.
    const u32 M = hdr->num_vertices;
    const u64 items = (u64)M * vpr;
    const int2* __restrict__ nb = reinterpret_cast<const int2*>(nbr_axis);
    const u32 stride = blocks * blockDim.x, dv = stride / vpr, dj = stride - dv * vpr;
    u64 e = (u64)block * blockDim.x + threadIdx.x;
    u32 v = (u32)e / vpr, j = (u32)e - v * vpr;   // item e is V j of vertex v's row (the first e fits 32 bits)
    int2 n = (v < M) ? load_once(nb + v) : make_int2(-1, -1);
    after_previous_kernel();
    if (hdr->status != 0) return;
    const V zero = {};
    auto rows = [&](auto once, auto mix) {
        while (e < items) {
            const V b = src[e];
            const V a = (n.x >= 0) ? src[(u64)n.x * vpr + j] : zero;
            const V c = (n.y >= 0) ? src[(u64)n.y * vpr + j] : zero;
            v += dv;
            j += dj;
            if (j >= vpr) {
                j -= vpr;
                v++;
            }
            if constexpr (decltype(once)::value) {
                if (v < M) n = load_once(nb + v);
            } else {
                if (v < M) n = __ldg(nb + v);
            }
            dst[e] = mix(a, b, c);
            e += stride;
        }
    };
    if constexpr (std::is_same<V, float4>::value) {
        if (items * lattices <= MOVED_ITEMS) {
            rows(std::true_type{}, [](V a, V b, V c) {
                float2 z = make_float2(0.f, 0.f);
                look_for_finite(z, a);
                look_for_finite(z, b);
                look_for_finite(z, c);
                return all_finite(z) ? mix_rows_moved(a, b, c) : mix_rows(a, b, c);
            });
            return;
        }
    }
    rows(std::is_same<V, double2>{}, [](V a, V b, V c) { return mix_rows(a, b, c); });
}
// blockIdx.y: the item, where one lattice serves several whose rows lie apart (item_v: V from one's rows to the next's).
template <typename V>
__global__ void __launch_bounds__(256, 8)
blur_axis(const Header* hdr, const int* __restrict__ nbr_axis, const V* __restrict__ src, V* __restrict__ dst, u32 vpr, u64 item_v) {
    blur_rows<V>(hdr, nbr_axis, src + blockIdx.y * item_v, dst + blockIdx.y * item_v, vpr, blockIdx.x, gridDim.x, gridDim.y);
}

// Two passes in one launch, along axes a and then b: a thread mixes the row that pass b needs of its vertex and of that one's
// two neighbours, from nine rows in all, and what pass a would have stored is rounded as it would have been: the same bits.
// All indices are older than the splat and are fetched before the wait, so that a pair of passes waits for rows once.  A
// pass of a lattice whose items (16 bytes of a row) fit the GPU's threads about once takes its launch and one round trip to
// L2, whatever it does; larger ones are bound by their rows, of which this reads half as many again.
// us a call: 4 x 180x240 x 3 59 -> 54, 512x512 x 3 in double, forward + backward, 185 -> 179, a CRF of 2 x 200x200 x 5 219 ->
// 189; 900 k vertices of one float4 239 -> 254, which is why it ends at PAIR_ITEMS (see blur_in_pairs).
// nbr_b null: pass a alone.  Four CTAs an SM, with five the mixes spill 64 bytes: 1024x1024 grey by RGB, forward + backward, 317.8 -> 312.0
// us, a CRF of 2 x 200x200 x 5 199.1 -> 189.2.
constexpr int PAIR_CTAS = 4;
constexpr u64 PAIR_ITEMS = 1000000, PAIR_ITEMS_WORST = 300000;   // by the bound, by one that is the worst case
template <typename V>
__device__ __forceinline__ void blur_pair_rows(const Header* hdr, const int* __restrict__ nbr_a, const int* __restrict__ nbr_b,
                                               const V* __restrict__ src, V* __restrict__ dst, u32 vpr, u32 block, u32 blocks) {
    const u32 M = hdr->num_vertices, items = M * vpr, stride = blocks * blockDim.x;
    const int2* __restrict__ na = reinterpret_cast<const int2*>(nbr_a);
    const int2* __restrict__ nb = reinterpret_cast<const int2*>(nbr_b);
    u32 e = block * blockDim.x + threadIdx.x, v = e / vpr, j = e - v * vpr;
    int u[3];      // the vertex and its neighbours along b
    int2 n[3];     // theirs along a
    auto look_up = [&]() {
        int2 beside = make_int2(-1, -1);
        if (v < M && nb) beside = load_once(nb + v);
        u[0] = v < M ? (int)v : -1;
        u[1] = beside.x;
        u[2] = beside.y;
#pragma unroll
        for (int k = 0; k < 3; k++) n[k] = u[k] >= 0 ? __ldg(na + u[k]) : make_int2(-1, -1);
    };
    look_up();
    after_previous_kernel();
    if (hdr->status != 0) return;
    const V zero = {};
    while (e < items) {
        V lo[3], mid[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            mid[k] = u[k] >= 0 ? src[(u32)u[k] * vpr + j] : zero;
            lo[k] = n[k].x >= 0 ? src[(u32)n[k].x * vpr + j] : zero;
            hi[k] = n[k].y >= 0 ? src[(u32)n[k].y * vpr + j] : zero;
        }
        float2 z = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            look_for_finite(z, lo[k]);
            look_for_finite(z, mid[k]);
            look_for_finite(z, hi[k]);
        }
        if (all_finite(z)) {   // (and so is what pass a makes of them)
#pragma unroll
            for (int k = 0; k < 3; k++) mid[k] = mix_rows_moved(lo[k], mid[k], hi[k]);
            if (nb) mid[0] = mix_rows_moved(mid[1], mid[0], mid[2]);
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) mid[k] = mix_rows(lo[k], mid[k], hi[k]);
            if (nb) mid[0] = mix_rows(mid[1], mid[0], mid[2]);
        }
        dst[e] = mid[0];
        e += stride;
        v = e / vpr;
        j = e - v * vpr;
        if (e < items) look_up();
    }
}
template <typename V>
__global__ void __launch_bounds__(256, PAIR_CTAS)
blur_pair(const Header* hdr, const int* __restrict__ nbr_a, const int* __restrict__ nbr_b, const V* __restrict__ src,
          V* __restrict__ dst, u32 vpr, u64 item_v) {
    blur_pair_rows<V>(hdr, nbr_a, nbr_b, src + blockIdx.y * item_v, dst + blockIdx.y * item_v, vpr, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------------------------
// slice_tiles (src/PermutohedralLatticeCPU.h:333-352: float multiply-then-add per remainder in
// ascending order, reciprocal of the homogeneous channel in double, one multiply per channel).
// Rows of one float4: slice_points, below.  Of wider ones the tile's are staged once in shared memory.
//
// Fast form (rows of VP floats, VP known at compile time; 8 to 32): one thread per point interpolates the whole
// row in registers (float4 reads of the cached rows, row stride padded against bank conflicts), the
// output block is assembled in shared memory and leaves by bulk asynchronous copies when its rows
// are 16-byte aligned.
// Generic form (any vd): a group of lanes per point, one float4 of channels per lane.
// ---------------------------------------------------------------------------------------------
template <int PD, int VP, int CT = 0>   // CT: see slice_tiles_fast
struct SliceFast {
    static constexpr int TP = Cfg<PD>::TP;
    static constexpr int RS = VP + 4;   // words between cached rows: 16-byte aligned, spreads banks
    // the output block ([TP][C], C < VP) reuses the space of the cached rows once every thread has read them
    __host__ __device__ static size_t region(int rows_cap) {
        const size_t rows = sizeof(float) * (size_t)rows_cap * RS, out = sizeof(float) * TP * VP;
        return rows > out ? rows : out;
    }
    static size_t bytes(int rows_cap) { return region(rows_cap) + sizeof(int) * TP; }
    // CTAs per SM asked of the compiler: what the row, the weights and the entry numbers of a point leave room for
    static constexpr int NEED = VP + 2 * (PD + 1);
    // With pd 2 and 3 the kernel waits for memory and not for shared memory's conflicts: a sixth CTA, 40 registers,
    // for rows that leave it room.  us a slice, six / five CTAs, by channels: 16 x 512x512, pd 2, 2.4 and 14.7 splats
    // an entry, 4 channels 106 / 102 and 76 / 83, 10 channels 141 / 159 and 94 / 106, 15 channels (8 bytes spilled)
    // 156 / 152 and 104 / 115, 19 channels 166 / 186 and 119 / 129, 21 channels, known at compile time (16 bytes),
    // 183 / 185 and 121 / 131; 4 x 64x128x128, pd 3, 1.3 and 6.6 splats, 4 channels 166 / 153 and 94 / 99, 10
    // channels 202 / 222 and 117 / 127, 15 channels (16 bytes) 268 / 237 and 125 / 126, 19 channels (12 bytes) 360 /
    // 331 and 134 / 148: tiles of few splats an entry lose up to an eighth, all others gain a tenth.  20 to 23
    // channels known at run time only would spill 48 bytes and gain nothing (2.4 splats 188 / 176).
    static constexpr bool SIX = (PD == 2 || PD == 3) && NEED <= (CT ? 30 : 28);
    static constexpr int CTAS = TP != 256 ? (VP > 24 ? 6 : 8) : SIX ? 6 : NEED <= 36 ? 5 : NEED <= 52 ? 4 : 3;
    static constexpr int ROWS_BYTES = (SIX ? 35 : 40) * 1024;   // of cached rows: so many CTAs fit the shared memory too
};

// The tile's vertex rows, `nrows` of them, on their way to shared memory.  CH copies per thread and trip: first the vertex
// numbers of all CH rows (independent loads, in flight together with the record loads before them), then the asynchronous
// copies that depend on them; interleaving them one by one would put a full memory latency between consecutive copies.
template <int PD, int VP>
__device__ __forceinline__ void stage_rows(float* rows_s, int nrows, const u32* __restrict__ list_ref, int base, const float4* v4) {
    constexpr int TP = Cfg<PD>::TP, QPR = VP / 4, RS = SliceFast<PD, VP>::RS, CH = 8;
    const int total = nrows * QPR;
    for (int i0 = threadIdx.x; i0 < total; i0 += CH * TP) {
        u32 vtx[CH];
#pragma unroll
        for (int c = 0; c < CH; c++) {
            const int i = i0 + c * TP;
            vtx[c] = (i < total) ? list_ref[base + i / QPR] : 0u;
        }
#pragma unroll
        for (int c = 0; c < CH; c++) {
            const int i = i0 + c * TP;
            if (i < total) {
                const int lrow = i / QPR, q = i - lrow * QPR;
                cp_async16(rows_s + lrow * RS + 4 * q, v4 + (size_t)vtx[c] * QPR + q);
            }
        }
    }
}

// A point's row: its pd + 1 vertex rows, weighted.
template <int PD, int VP>
__device__ __forceinline__ void mix_rows_of_point(float (&acc)[VP], bool valid, const int (&l)[PD + 1], const float (&w)[PD + 1],
                                                  const float* rows_s, int nrows, int cnt, int rows_cap,
                                                  const u32* __restrict__ list_ref, int base, const float4* v4) {
    constexpr int QPR = VP / 4, RS = SliceFast<PD, VP>::RS;
#pragma unroll
    for (int j = 0; j < VP; j++) acc[j] = 0.f;
    if (valid && cnt <= rows_cap) {
        // every row of the tile is cached (the usual case): plain shared-memory reads
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const float4* row = reinterpret_cast<const float4*>(rows_s + l[r] * RS);
#pragma unroll
            for (int q = 0; q < QPR; q++) {
                const float4 x = row[q];
                acc[4 * q] = PL_FADD(acc[4 * q], PL_FMUL(w[r], x.x));
                acc[4 * q + 1] = PL_FADD(acc[4 * q + 1], PL_FMUL(w[r], x.y));
                acc[4 * q + 2] = PL_FADD(acc[4 * q + 2], PL_FMUL(w[r], x.z));
                acc[4 * q + 3] = PL_FADD(acc[4 * q + 3], PL_FMUL(w[r], x.w));
            }
        }
    } else if (valid) {
        // a tile with more entries than the cache holds: the rest comes straight from global memory
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const float4* row = (l[r] < nrows) ? reinterpret_cast<const float4*>(rows_s + l[r] * RS)
                                               : v4 + (size_t)list_ref[base + l[r]] * QPR;
#pragma unroll
            for (int q = 0; q < QPR; q++) {
                const float4 x = row[q];
                acc[4 * q] = PL_FADD(acc[4 * q], PL_FMUL(w[r], x.x));
                acc[4 * q + 1] = PL_FADD(acc[4 * q + 1], PL_FMUL(w[r], x.y));
                acc[4 * q + 2] = PL_FADD(acc[4 * q + 2], PL_FMUL(w[r], x.z));
                acc[4 * q + 3] = PL_FADD(acc[4 * q + 3], PL_FMUL(w[r], x.w));
            }
        }
    }
}

// CT: the channels where they are fixed at compile time, else 0 (VP - 4 <= C < VP, a few registers more).
template <int PD, int VP, int CT>
__global__ void __launch_bounds__(Cfg<PD>::TP, SliceFast<PD, VP, CT>::CTAS)
slice_tiles_fast(Geom g, float* __restrict__ output, const Header* hdr, const int2* __restrict__ tile_info,
                 const u16* __restrict__ rec, const float* __restrict__ rec_w,
                 const u32* __restrict__ list_ref, const float* __restrict__ vsrc, int channels, int rows_cap, int bulk_ok,
                 Watch watch) {
    // Launched to overlap the tail of the last blur pass: the status word, the tile's range and the per-point
    // records are older than any blur pass and are fetched before the wait; the vertex rows after it.
    const int C = CT ? CT : channels;
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, QPR = VP / 4;
    constexpr int RS = SliceFast<PD, VP>::RS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* rows_s = reinterpret_cast<float*>(smem_raw);                                         // [rows_cap][RS]
    float* out_s = reinterpret_cast<float*>(smem_raw);                                          // [TP][C], later
    int* prow_s = reinterpret_cast<int*>(smem_raw + SliceFast<PD, VP>::region(rows_cap));       // [TP]
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile;
    const u32 status = hdr->status;   // final by now, the same in every thread; one round trip with all that follows
    const int2 info = tile_info[tile];
    const int base = info.x + first_entry_of<PD>(g, tpos.item), cnt = info.y;
    const int nrows = min(cnt, rows_cap);
    const float4* v4 = reinterpret_cast<const float4*>(vsrc);
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    float w[PD + 1];
    int l[PD + 1];
    const u16* rec_tile = rec + (size_t)tile * SPLATS;
    const float* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        l[r] = valid ? load_record<PD>(rec_tile + r * TP + tid) : 0;
        w[r] = valid ? load_record<PD>(recw_tile + r * TP + tid) : 0.f;
    }
    if (status != 0) {
        poison_tile_output(g, output, C);
        report_late(watch, hdr);
        wait_for_previous_kernel();
        return;
    }
    wait_for_previous_kernel();
    stage_rows<PD, VP>(rows_s, nrows, list_ref, base, v4);
    cp_async_wait_all();
    __syncthreads();
    float acc[VP];
    mix_rows_of_point<PD, VP>(acc, valid, l, w, rows_s, nrows, cnt, rows_cap, list_ref, base, v4);
    __syncthreads();   // every cached row has been read: the output block may overwrite them
    if (valid) {
        const int last = C - (VP - 4);   // channels in the row's last quad; the next one is the homogeneous channel
        const float norm = last == 0 ? acc[VP - 4] : last == 1 ? acc[VP - 3] : last == 2 ? acc[VP - 2] : acc[VP - 1];
        const float inv = (float)(1.0 / (double)norm);
        float* o = out_s + tid * C;
        if (last == 0) {   // whole quads: rows a multiple of 16 bytes long would collide on banks as single floats
#pragma unroll
            for (int j = 0; j < VP - 4; j += 4)
                *reinterpret_cast<float4*>(o + j) = make_float4(PL_FMUL(acc[j], inv), PL_FMUL(acc[j + 1], inv),
                                                                PL_FMUL(acc[j + 2], inv), PL_FMUL(acc[j + 3], inv));
        } else {
#pragma unroll
            for (int j = 0; j < VP - 4; j++) o[j] = PL_FMUL(acc[j], inv);
#pragma unroll
            for (int j = 0; j < 3; j++)
                if (j < last) o[VP - 4 + j] = PL_FMUL(acc[VP - 4 + j], inv);
        }
    }
    if (bulk_ok) {
        fence_async_proxy();
        __syncthreads();
        if (tid < g.TY) {
            int first, count;
            if (tile_row(g, this_tile(g), tid, first, count))   // recomputed: keeps registers free above
                bulk_store(output + (size_t)first * C, out_s + (size_t)tid * g.TX * C, (unsigned)count * C * 4u);
            bulk_store_finish();
        }
    } else {
        __syncthreads();
        // element k = tid, tid + TP, ... is channel j of point p; (p, j) advance without a division
        const int DP = TP / C, DJ = TP - DP * C;
        int p = tid / C, j = tid - p * C;
        for (int k = tid; k < TP * C; k += TP) {
            const int row = prow_s[p];
            if (row >= 0) output[(size_t)row * C + j] = out_s[k];
            p += DP;
            j += DJ;
            if (j >= C) {
                j -= C;
                p++;
            }
        }
    }
}

// Rows of one float4: a thread a point, straight from the rows in global memory.  A tile's rows are a kilobyte or a few,
// which L1 holds as well as shared memory would, and without the copies, the barriers around them and the 40 KB a CTA
// that left an SM with fewer than half its warps.  Two volumes of 111x128x120 points, 2 channels: 69 -> 36 us; 800x1200 x 3,
// pd 5: 24 -> 18; 1 M points, pd 16: 92 -> 60.
__device__ __forceinline__ float4 load_row(const float4* p) {   // never moved ahead of the wait for the kernel before
    float4 x;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                 : "l"(p)
                 : "memory");
    return x;
}
template <int PD, int C>
// (CTAs an SM: left alone the compiler takes up to 91 registers at pd 16; 8 M points there 0.46 / 0.41 ms)
__global__ void __launch_bounds__(Cfg<PD>::TP, Cfg<PD>::COMPACT || (PD == 5 && C > 1) ? 7 : PD > 5 ? 5 : 8)
slice_points(Geom g, float* __restrict__ output, const Header* hdr, const int2* __restrict__ tile_info,
             const u16* __restrict__ rec, const float* __restrict__ rec_w, const u32* __restrict__ list_ref,
             const float* __restrict__ vsrc, Watch watch) {
    // (what is read before the wait is older than any blur pass, as in slice_tiles_fast)
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS;
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x;
    const u32 status = hdr->status;   // final by now: the same in every thread
    const int base = tile_info[tpos.tile].x + first_entry_of<PD>(g, tpos.item);
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    auto stop = [&]() {
        poison_tile_output(g, output, C);
        report_late(watch, hdr);
        wait_for_previous_kernel();
    };
    if (Cfg<PD>::COMPACT && status != 0) return stop();
    const size_t at = (size_t)tpos.tile * SPLATS + tid;
    float w[PD + 1];
    u32 v[PD + 1];
#pragma unroll
    for (int r = 0; r <= PD; r++) v[r] = valid ? load_record<PD>(rec + at + r * TP) : 0;
#pragma unroll
    for (int r = 0; r <= PD; r++) w[r] = valid ? load_record<PD>(rec_w + at + r * TP) : 0.f;
    if (!Cfg<PD>::COMPACT && status != 0) return stop();
    const u32* ref = list_ref + base;
#pragma unroll
    for (int r = 0; r <= PD; r++) v[r] = valid ? ref[v[r]] : 0u;
    wait_for_previous_kernel();
    if (!valid) return;
    const float4* v4 = reinterpret_cast<const float4*>(vsrc);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        const float4 x = load_row(v4 + v[r]);
        acc.x = PL_FADD(acc.x, PL_FMUL(w[r], x.x));
        acc.y = PL_FADD(acc.y, PL_FMUL(w[r], x.y));
        acc.z = PL_FADD(acc.z, PL_FMUL(w[r], x.z));
        acc.w = PL_FADD(acc.w, PL_FMUL(w[r], x.w));
    }
    const float inv = (float)(1.0 / (double)(C == 1 ? acc.y : C == 2 ? acc.z : acc.w));
    float* o = output + ((size_t)item * g.n + pix) * C;
    store_once(o, PL_FMUL(acc.x, inv));
    if constexpr (C > 1) store_once(o + 1, PL_FMUL(acc.y, inv));
    if constexpr (C > 2) store_once(o + 2, PL_FMUL(acc.z, inv));
}

template <int PD>
struct SliceCfg {
    static constexpr int PW = ((2 * (PD + 1) + 1 + 3) / 4) * 4;   // words of a point record
};

template <int PD>
__global__ void __launch_bounds__(Cfg<PD>::TP)
slice_tiles_generic(Geom g, float* __restrict__ output, const Header* hdr, const int2* __restrict__ tile_info,
                    const u16* __restrict__ rec, const float* __restrict__ rec_w,
                    const u32* __restrict__ list_ref, const float* __restrict__ vsrc, int vd, int rows_cap, Watch watch) {
    wait_for_previous_kernel();
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, PW = SliceCfg<PD>::PW;
    const int C = vd - 1, VP = padded_vd(vd), QPR = VP >> 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4* rows4 = reinterpret_cast<float4*>(smem_raw);                            // [rows_cap][QPR]
    float* prec_s = reinterpret_cast<float*>(rows4 + (size_t)rows_cap * QPR);       // [TP][PW]
    int* prow_s = reinterpret_cast<int*>(prec_s + (size_t)TP * PW);                 // [TP]
    if (call_failed(hdr)) {
        poison_tile_output(g, output, C);
        report_late(watch, hdr);
        return;
    }
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile, lane = tid & 31, warp = tid >> 5;
    const int2 info = tile_info[tile];
    const int base = info.x + first_entry_of<PD>(g, tpos.item), cnt = info.y;
    const int nrows = min(cnt, rows_cap);
    const float4* v4 = reinterpret_cast<const float4*>(vsrc);
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    float w[PD + 1];
    int l[PD + 1];
    const u16* rec_tile = rec + (size_t)tile * SPLATS;
    const float* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        l[r] = valid ? load_record<PD>(rec_tile + r * TP + tid) : 0;
        w[r] = valid ? load_record<PD>(recw_tile + r * TP + tid) : 0.f;
    }
    {   // row staging: vertex numbers of CH rows first, then the copies that depend on them (see slice_tiles_fast)
        constexpr int CH = 8;
        const int total = nrows * QPR;
        for (int i0 = tid; i0 < total; i0 += CH * TP) {
            u32 vtx[CH];
#pragma unroll
            for (int c = 0; c < CH; c++) {
                const int i = i0 + c * TP;
                vtx[c] = (i < total) ? list_ref[base + i / QPR] : 0u;
            }
#pragma unroll
            for (int c = 0; c < CH; c++) {
                const int i = i0 + c * TP;
                if (i < total) cp_async16(rows4 + i, v4 + (size_t)vtx[c] * QPR + (i - (i / QPR) * QPR));
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (valid) {
        const float* rows = reinterpret_cast<const float*>(rows4);
        float norm = 0.f;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const float hv = (l[r] < nrows) ? rows[l[r] * VP + C]
                                            : vsrc[(size_t)list_ref[base + l[r]] * VP + C];
            norm = PL_FADD(norm, PL_FMUL(w[r], hv));
        }
        float* pr = prec_s + tid * PW;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            pr[r] = w[r];
            pr[PD + 2 + r] = __int_as_float(l[r]);
        }
        pr[PD + 1] = (float)(1.0 / (double)norm);
    }
    __syncthreads();

    const LaneMap lm(QPR, lane);
    if (!lm.active) return;
    for (int i = lm.g; i < 32; i += lm.ppw) {
        const int p = warp * 32 + i;
        const int row = prow_s[p];
        if (row < 0) continue;
        float pr[PW];
        const float4* pr4 = reinterpret_cast<const float4*>(prec_s + p * PW);
#pragma unroll
        for (int k = 0; k < PW / 4; k++) {
            const float4 t = pr4[k];
            pr[4 * k] = t.x; pr[4 * k + 1] = t.y; pr[4 * k + 2] = t.z; pr[4 * k + 3] = t.w;
        }
        const float inv = pr[PD + 1];
        const float4* rp[PD + 1];
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int lr = __float_as_int(pr[PD + 2 + r]);
            rp[r] = (lr < nrows) ? (rows4 + lr * QPR) : (v4 + (size_t)list_ref[base + lr] * QPR);
        }
        float* out_row = output + (size_t)row * C;
        for (int q = lm.q0; q < QPR; q += lm.gs) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int r = 0; r <= PD; r++) {
                const float4 x = rp[r][q];
                acc.x = PL_FADD(acc.x, PL_FMUL(pr[r], x.x));
                acc.y = PL_FADD(acc.y, PL_FMUL(pr[r], x.y));
                acc.z = PL_FADD(acc.z, PL_FMUL(pr[r], x.z));
                acc.w = PL_FADD(acc.w, PL_FMUL(pr[r], x.w));
            }
            const int j = 4 * q;
            if (j < C) out_row[j] = PL_FMUL(acc.x, inv);
            if (j + 1 < C) out_row[j + 1] = PL_FMUL(acc.y, inv);
            if (j + 2 < C) out_row[j + 2] = PL_FMUL(acc.z, inv);
            if (j + 3 < C) out_row[j + 3] = PL_FMUL(acc.w, inv);
        }
    }
}

}  // namespace pl
