// T = double: splat, blur and slice over rows of doubles.  The lattice structure (keys, table,
// vertex and neighbour tables) comes from the same kernels as for float; only the geometry
// arithmetic and the value rows differ.
#pragma once
#include "common.cuh"
#include "splat.cuh"

namespace pl {

// Doubles of a vertex row: vd padded to a multiple of 2 (16-byte rows).
__host__ __device__ __forceinline__ int padded_vd_f64(int vd) { return (vd + 1) & ~1; }

// Lanes that share a row (a splat's window, a point of the slice), as a logarithm: the power of two that holds
// `pairs` double2, at most a warp.
__device__ __forceinline__ int lanes_log2_f64(int pairs) {
    return pairs > 16 ? 5 : pairs > 8 ? 4 : pairs > 4 ? 3 : pairs > 2 ? 2 : pairs > 1 ? 1 : 0;
}

// Doubles of a row that the splat stages and sums at a time: 64 KB of input for a tile of 256 points.
constexpr int SPLAT64_BLOCK = 32;

template <int PD>
struct Splat64 {
    static constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, SORTED = Cfg<PD>::SREC;
    static size_t bytes(int vd) {
        const int vp = padded_vd_f64(vd), staged = vp < SPLAT64_BLOCK ? vp : SPLAT64_BLOCK;
        return sizeof(double) * TP * staged + sizeof(uint4) * SORTED + sizeof(int) * SPLATS + sizeof(int) * TP;
    }
};

// V[vertex] += sum over the tile's splats of weight * [input channels, 1]
// (src/PermutohedralLatticeCPU.h:306-313).  As splat_tiles_rows: the tile's splats are counting-sorted by entry and
// cut into windows, a group of lanes with a double2 of the row each walks a window and sums each entry's run in
// registers, the input rows lie in shared memory (channel C as 1, padding as 0), SPLAT64_BLOCK doubles at a time.
// Bound by the latency of the serial walk; a warp per window with a channel per lane, as before, left 28 of its
// 32 lanes idle on an RGB image.  512 x 512 RGB,
// forward + backward: 475 -> 225 us for this kernel and the slice together; this one now takes 21 us a call.
template <int PD>
__global__ void __launch_bounds__(Cfg<PD>::TP)
splat_tiles_f64(Geom g, const double* __restrict__ input, Header* hdr, const int2* __restrict__ tile_info,
                const u16* __restrict__ rec, const double* __restrict__ rec_w,
                const u32* __restrict__ list_ref, double* __restrict__ v0, int vd) {
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, WL = Cfg<PD>::WL;
    const int C = vd - 1, VP = padded_vd_f64(vd), SP = min(VP, SPLAT64_BLOCK);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* in_s = reinterpret_cast<double*>(smem_raw);                        // [TP][SP]
    uint4* sorted_s = reinterpret_cast<uint4*>(in_s + (size_t)TP * SP);        // [SORTED]
    int* cur_s = reinterpret_cast<int*>(sorted_s + Splat64<PD>::SORTED);       // [SPLATS]
    int* prow_s = cur_s + SPLATS;                                              // [TP]
    __shared__ int wsum_s[32];
    // Launched to overlap the tail of link_neighbours, as splat_tiles_rows is: the input and the records are older.
    if (call_failed(hdr)) {
        wait_for_previous_kernel();
        return;
    }
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile;
    const int2 info = tile_info[tile];
    const int base = info.x, nloc = info.y;
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    for (int i = tid; i < nloc; i += TP) cur_s[i] = 0;
    int l[PD + 1];
    double w[PD + 1];
    const u16* rec_tile = rec + (size_t)tile * SPLATS;
    const double* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        l[r] = valid ? rec_tile[r * TP + tid] : 0;
        w[r] = valid ? recw_tile[r * TP + tid] : 0.0;
    }
    const int total = __syncthreads_count(valid) * (PD + 1);

    for (int j0 = 0; j0 < VP; j0 += SPLAT64_BLOCK) {
        const int width = min(SPLAT64_BLOCK, VP - j0), chans = min(width, C - j0);   // of this block; input channels of it
        if (j0 > 0) __syncthreads();   // the block before has been read
        if (chans > 0) {
            // element k = tid, tid + TP, ... is channel j of point p; (p, j) advance without a division
            const int dp = TP / chans, dj = TP - dp * chans;
            int p = tid / chans, j = tid - p * chans;
            for (int k = tid; k < TP * chans; k += TP) {
                const int row = prow_s[p];
                if (row >= 0) cp_async8(in_s + p * width + j, input + (size_t)row * C + j0 + j);
                p += dp;
                j += dj;
                if (j >= chans) {
                    j -= chans;
                    p++;
                }
            }
        }
        for (int j = max(chans, 0); j < width; j++) in_s[tid * width + j] = (j0 + j == C) ? 1.0 : 0.0;
        if (j0 == 0) SplatCommon<PD>::template sort_splats<WL>(valid, l, w, nloc, sorted_s, cur_s, wsum_s);
        cp_async_wait_all();
        if (j0 == 0) {
            wait_for_previous_kernel();     // from here on the entries' vertices and the zeroed rows
            if (call_failed(hdr)) return;   // a failure of the index stage
        }
        __syncthreads();

        const int pairs = width >> 1, lw_log2 = lanes_log2_f64(pairs);
        const int h = tid & ((1 << lw_log2) - 1), wl = (PD + 1) << lw_log2;
        const int first = (tid >> lw_log2) * wl, end = min(first + wl, total);
        if (first >= end || h >= pairs) continue;
        const double2* in2 = reinterpret_cast<const double2*>(in_s) + h;
        const int ch = j0 + 2 * h;   // this lane's channels: ch, ch + 1 (the last one may be padding)
        double2 acc = make_double2(0.0, 0.0);
        int cur = (int)(sorted_s[Cfg<PD>::srec_slot(first)].x >> 16);
        u32 vcur = list_ref[base + cur];
        for (int pos = first; pos < end; pos += WL) {
            const uint4* sp = sorted_s + Cfg<PD>::srec_slot(pos);
            const int count = min(WL, end - pos);
#pragma unroll 4
            for (int i = 0; i < count; i++) {
                const uint4 pw = sp[i];
                const int e = (int)(pw.x >> 16);
                if (e != cur) {
                    double* row = v0 + (size_t)vcur * VP + ch;
                    red_add_f64(row, acc.x);
                    if (ch < C) red_add_f64(row + 1, acc.y);
                    acc = make_double2(0.0, 0.0);
                    cur = e;
                    vcur = list_ref[base + cur];
                }
                const double wt = __hiloint2double((int)pw.w, (int)pw.z);
                const double2 x = in2[(pw.x & 0xFFFFu) * pairs];
                acc.x = __fma_rn(wt, x.x, acc.x);
                acc.y = __fma_rn(wt, x.y, acc.y);
            }
        }
        double* row = v0 + (size_t)vcur * VP + ch;
        red_add_f64(row, acc.x);
        if (ch < C) red_add_f64(row + 1, acc.y);
    }
}

// Slice (src/PermutohedralLatticeCPU.h:333-352): per point and channel the weighted sum over the
// remainders in ascending order, then one multiply by the reciprocal of the homogeneous channel.
// A group of lanes per point, a double2 of the row each (rows beyond a warp's 32 are walked 32 at a time); the
// homogeneous sum comes from the lane that holds its channel.  The rows are read through L1, where neighbouring
// points share them.  A warp per point with a channel per lane, as before, left most lanes idle and every lane
// summed the homogeneous channel again.  Its figure
// stands at splat_tiles_f64; it takes 11 us a call now.
template <int PD>
__global__ void __launch_bounds__(Cfg<PD>::TP)
slice_tiles_f64(Geom g, double* __restrict__ output, const Header* hdr, const int2* __restrict__ tile_info,
                const u16* __restrict__ rec, const double* __restrict__ rec_w,
                const u32* __restrict__ list_ref, const double* __restrict__ vsrc, int vd, Watch watch) {
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS;
    const int C = vd - 1, VP = padded_vd_f64(vd), pairs = VP >> 1;
    __shared__ double w_s[SPLATS];
    __shared__ u32 v_s[SPLATS];
    __shared__ int prow_s[TP];
    if (call_failed(hdr)) {
        poison_tile_output(g, output, C);
        report_late(watch, hdr);
        wait_for_previous_kernel();
        return;
    }
    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile, lane = tid & 31, warp = tid >> 5;
    const int base = tile_info[tile].x;
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    const u16* rec_tile = rec + (size_t)tile * SPLATS;
    const double* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        w_s[r * TP + tid] = valid ? recw_tile[r * TP + tid] : 0.0;
        v_s[r * TP + tid] = valid ? list_ref[base + rec_tile[r * TP + tid]] : 0u;
    }
    wait_for_previous_kernel();   // the last blur pass: all that was read up to here is older
    __syncwarp();   // a warp reads the points its own lanes have written
    const int lw_log2 = lanes_log2_f64(pairs), lw = 1 << lw_log2;
    const int h = lane & (lw - 1), group = lane >> lw_log2;
    const double2* __restrict__ v2 = reinterpret_cast<const double2*>(vsrc);
    const int hom = (C >> 1) & (lw - 1);   // lane of the group that meets the homogeneous channel
    for (int i = group; i < 32; i += 32 >> lw_log2) {
        const int p = warp * 32 + i;
        const int row = prow_s[p];
        double inv = 0.0;
        // all lanes of a warp make the same trips: the shuffle below needs every one of them; the last quad of the
        // row, with the homogeneous channel, is taken first
        for (int q0 = (pairs - 1) & ~(lw - 1); q0 >= 0; q0 -= lw) {
            const int q = q0 + h;
            double2 acc = make_double2(0.0, 0.0);
            if (row >= 0 && q < pairs) {
#pragma unroll
                for (int r = 0; r <= PD; r++) {
                    const double w = w_s[r * TP + p];
                    const double2 x = __ldg(v2 + (size_t)v_s[r * TP + p] * pairs + q);
                    acc.x = PL_DADD(acc.x, PL_DMUL(w, x.x));
                    acc.y = PL_DADD(acc.y, PL_DMUL(w, x.y));
                }
            }
            if (q0 + lw >= pairs) {
                const double norm = __shfl_sync(0xFFFFFFFFu, (C & 1) ? acc.y : acc.x, hom, lw);
                inv = __ddiv_rn(1.0, norm);
            }
            if (row >= 0 && q < pairs) {
                double* o = output + (size_t)row * C + 2 * q;
                if (2 * q < C) o[0] = PL_DMUL(acc.x, inv);
                if (2 * q + 1 < C) o[1] = PL_DMUL(acc.y, inv);
            }
        }
    }
}

}  // namespace pl
