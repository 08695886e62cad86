// The pointwise half of a dense-CRF mean-field update, fused into one pass over memory:
//   q_out = softmax over labels of ( -unaries - (wb * q_bilateral + ws * q_spatial) @ compatibility ).
// The two filtered label distributions come from the lattice filter (appearance and smoothness kernels);
// this kernel replaces the scale, add, matrix product, subtraction and softmax passes that would each
// read and write all points x labels floats.  The reference library ships no CRF code (its README names
// CRF-as-RNN as its user), so this follows the published mean-field update, not a reference file.
#pragma once
#include "common.cuh"
#include "splat.cuh"
#include "blur_slice.cuh"

namespace pl {

// Row stride of the shared-memory tiles: odd, so that threads reading their own point's row never share a bank.
__host__ __device__ __forceinline__ int crf_row_stride(int L) { return L | 1; }

__host__ __forceinline__ size_t crf_smem_bytes(int tpb, int L) {
    return sizeof(float) * ((size_t)2 * tpb * crf_row_stride(L) + (size_t)L * L);
}

// One CTA per TPB consecutive points, whose [point][label] blocks are contiguous in memory: the block is
// loaded with coalesced accesses (message and negated unaries formed on the way), then one thread per
// point does the L x L product, the softmax, and the block leaves the same way it came.
// compat == nullptr: Potts model (1 - identity): pairwise_k = sum_j m_j - m_k.
// LT > 0: Potts model with the label count fixed at compile time (a point's rows then live in registers:
// one shared-memory read and one write per value); LT == 0: any count, any compatibility (rows stay in
// shared memory).
// qb == nullptr: no message yet, the distributions that an inference starts from (softmax of -unaries; as torch
// operations a negation and a softmax, 21 us on 375x500 x 21, so 11).
template <int TPB, int LT>
__global__ void __launch_bounds__(TPB)
crf_update(float* __restrict__ q_out, const float* __restrict__ unaries, const float* __restrict__ qb,
           const float* __restrict__ qs, const float* __restrict__ compat, float wb, float ws,
           long long n_points, int L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int LS = crf_row_stride(L);
    float* m_s = reinterpret_cast<float*>(smem_raw);   // [TPB][LS] message, later the result
    float* z_s = m_s + (size_t)TPB * LS;               // [TPB][LS] -unaries, later the logits
    float* c_s = z_s + (size_t)TPB * LS;               // [L][L]
    const int tid = threadIdx.x;
    const long long p0 = (long long)blockIdx.x * TPB;
    const int np = (int)min((long long)TPB, n_points - p0);
    const int total = np * L;
    const size_t g0 = (size_t)p0 * L;
    if (compat)
        for (int i = tid; i < L * L; i += TPB) c_s[i] = compat[i];
    // element e = tid, tid + TPB, ... is label j of point p; (p, j) advance without a division
    const int DP = TPB / L, DJ = TPB % L;
    {
        int p = tid / L, j = tid - p * L;
        for (int e = tid; e < total; e += TPB) {
            m_s[p * LS + j] = qb ? PL_FADD(PL_FMUL(wb, qb[g0 + e]), PL_FMUL(ws, qs[g0 + e])) : 0.f;
            z_s[p * LS + j] = -unaries[g0 + e];
            p += DP;
            j += DJ;
            if (j >= L) {
                j -= L;
                p++;
            }
        }
    }
    __syncthreads();
    if (tid < np) {
        float* m = m_s + tid * LS;
        float* z = z_s + tid * LS;
        if constexpr (LT > 0) {
            float mr[LT], zr[LT];
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < LT; j++) {
                mr[j] = m[j];
                zr[j] = z[j];
                sum = PL_FADD(sum, mr[j]);
            }
            float mx = -INFINITY;
#pragma unroll
            for (int k = 0; k < LT; k++) {
                zr[k] = PL_FADD(zr[k], -PL_FADD(sum, -mr[k]));
                mx = fmaxf(mx, zr[k]);
            }
            float den = 0.f;
#pragma unroll
            for (int k = 0; k < LT; k++) {
                zr[k] = expf(PL_FADD(zr[k], -mx));
                den = PL_FADD(den, zr[k]);
            }
            const float inv = PL_FDIV(1.f, den);
#pragma unroll
            for (int k = 0; k < LT; k++) m[k] = PL_FMUL(zr[k], inv);
        } else {
            float mx = -INFINITY;
            if (compat) {
                for (int k = 0; k < L; k++) {
                    float pair = 0.f;
                    for (int j = 0; j < L; j++) pair = PL_FMA(m[j], c_s[j * L + k], pair);
                    const float zk = PL_FADD(z[k], -pair);
                    z[k] = zk;
                    mx = fmaxf(mx, zk);
                }
            } else {
                float sum = 0.f;
                for (int j = 0; j < L; j++) sum = PL_FADD(sum, m[j]);
                for (int k = 0; k < L; k++) {
                    const float zk = PL_FADD(z[k], -PL_FADD(sum, -m[k]));
                    z[k] = zk;
                    mx = fmaxf(mx, zk);
                }
            }
            float den = 0.f;
            for (int k = 0; k < L; k++) {
                const float ex = expf(PL_FADD(z[k], -mx));
                m[k] = ex;
                den = PL_FADD(den, ex);
            }
            const float inv = PL_FDIV(1.f, den);
            for (int k = 0; k < L; k++) m[k] = PL_FMUL(m[k], inv);
        }
    }
    __syncthreads();
    {
        int p = tid / L, j = tid - p * L;
        for (int e = tid; e < total; e += TPB) {
            q_out[g0 + e] = m_s[p * LS + j];
            p += DP;
            j += DJ;
            if (j >= L) {
                j -= L;
                p++;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// A whole mean-field step of a CRF whose two lattices, appearance (A) and smoothness (S), have tiles of the same points:
// each stage of both in one launch (the blur passes of large lattices one after the other), and the update in the slice.  On one image the stages are small kernels, bound by their
// launches and by nearly empty last waves: apart, a step is 17 launches, and the filtered distributions go through memory
// once more each way.  375x500 x 21: 98 -> 66 us a step; 2 x 200x200 x 5, five steps and both builds, 360 -> 191; 16 x 512x512 x 21 1187 -> 964,
// 16 x 512x512 x 8 864 -> 800, 8 x 512x512 x 21 of noisy images 2013 -> 1872, 2000x3000 x 10 1988 -> 1869.
// ---------------------------------------------------------------------------------------------
struct LatticeRows {   // a kept lattice, as its workspace holds it
    Header* hdr;
    const int2* tile_info;
    const u16* rec;
    const float* rec_w;
    const uint2* srec;
    const u32* list_ref;
    const int* nbr;
    u64 max_entries;
    float *v0, *v1;
};

__global__ void __launch_bounds__(256)
crf_zero_rows(LatticeRows a, LatticeRows s, u32 quads /* of a row */) {
    after_previous_kernel();
    const LatticeRows& l = blockIdx.y ? s : a;
    if (l.hdr->status != 0) return;
    const u64 items = (u64)l.hdr->num_vertices * quads;
    float4* rows = reinterpret_cast<float4*>(l.v0);
    for (u64 i = (u64)blockIdx.x * 256 + threadIdx.x; i < items; i += (u64)gridDim.x * 256)
        rows[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Tile grid of one lattice, twice: first every tile of A, whose tiles take longer, then those of S.
template <int PDA, int PDS, int VD>
__global__ void __launch_bounds__(Cfg<PDA>::TP, 5)
crf_splat(Geom g, const float* __restrict__ input, LatticeRows a, LatticeRows s, int vd, int bulk_ok) {
    const int tiles = g.grid3 ? (int)gridDim.z / 2 : (int)gridDim.x / 2, here = g.grid3 ? blockIdx.z : blockIdx.x;
    const bool second = here >= tiles;
    const int mine = second ? here - tiles : here;
    const TilePos tpos = tile_at(g, g.grid3 ? (int)blockIdx.x : mine, mine);
    if (!second)
        splat_rows<PDA, VD, true, FloatSum, float>(g, tpos, input, a.hdr, a.tile_info, a.rec, a.rec_w, a.srec, a.list_ref, a.v0, vd, bulk_ok);
    else
        splat_rows<PDS, VD, true, FloatSum, float>(g, tpos, input, s.hdr, s.tile_info, s.rec, s.rec_w, s.srec, s.list_ref, s.v0, vd, bulk_ok);
}

// Passes 2 `pair` and 2 pair + 1 of both (S: as many as it has; see blur_pair_rows), from v0 to v1 in even pairs.
template <int PDA, int PDS>
__global__ void __launch_bounds__(256, PAIR_CTAS)
crf_blur_pair(LatticeRows a, LatticeRows s, int only, int pair, u32 quads) {
    const bool second = only ? only == 2 : blockIdx.y != 0;
    const LatticeRows& l = second ? s : a;
    const float4* src = reinterpret_cast<const float4*>((pair & 1) ? l.v1 : l.v0);
    float4* dst = reinterpret_cast<float4*>((pair & 1) ? l.v0 : l.v1);
    const int* nbr = l.nbr + 4 * (u64)pair * l.max_entries;
    blur_pair_rows<float4>(l.hdr, nbr, 2 * pair + 1 <= (second ? PDS : PDA) ? nbr + 2 * l.max_entries : nullptr, src, dst, quads, blockIdx.x, gridDim.x);
}

// A pass of both, blockIdx.y 0 and 1.  (The fields of each by themselves; choosing between two LatticeRows spilled 40 bytes in place of
// 8: 8 x 512x512 x 21 of noisy images 2266 -> 2076 us a step.)
__global__ void __launch_bounds__(256, 8)
crf_blur(const Header* hdr_a, const int* nbr_a, const float4* src_a, float4* dst_a, const Header* hdr_s, const int* nbr_s,
         const float4* src_s, float4* dst_s, u32 quads) {
    const bool second = blockIdx.y != 0;
    blur_rows<float4>(second ? hdr_s : hdr_a, second ? nbr_s : nbr_a, second ? src_s : src_a, second ? dst_s : dst_a, quads,
            blockIdx.x, gridDim.x, 1);
}

// Both slices and the update of a Potts model (see crf_update, whose arithmetic this is).  A thread a point: the tile's rows
// of A are staged, mixed and normalised, then those of S in the same memory, while the unaries arrive; the message and
// the logits stay in registers: 80 of them, for three CTAs an SM; from rows of 16 floats on 4 to 92 bytes are spilled (48 at 21 labels).
template <int PDA, int PDS, int VP>
struct CrfSlices {
    static constexpr int TP = Cfg<PDA>::TP, RS = VP + 4;
    static constexpr int ROWS = 40 * 1024 / (4 * RS) < Cfg<PDA>::SPLATS ? 40 * 1024 / (4 * RS) : Cfg<PDA>::SPLATS;
    static constexpr size_t REGION = sizeof(float) * (ROWS * RS > TP * VP ? ROWS * RS : TP * VP);
    __host__ __device__ static constexpr int stride(int labels) { return labels | 1; }   // of the unaries in shared memory
    __host__ __device__ static constexpr size_t bytes(int labels) {
        return REGION + ((sizeof(float) * TP * stride(labels) + 15) & ~(size_t)15) + sizeof(int) * TP;
    }
    static_assert(Cfg<PDA>::TP == Cfg<PDS>::TP && SliceFast<PDA, VP>::RS == RS && SliceFast<PDS, VP>::RS == RS, "one staging area");
};
template <int PD, int VP>
__device__ __forceinline__ void slice_message(float (&m)[VP], float weight, bool first, const TilePos& tpos, bool valid,
                                              const LatticeRows& lat, const float* v, float* rows_s, int rows_cap, int C) {
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS;
    const int2 info = lat.tile_info[tpos.tile];
    const int nrows = min(info.y, rows_cap);
    float w[PD + 1];
    int l[PD + 1];
    const u16* rec_tile = lat.rec + (size_t)tpos.tile * SPLATS + threadIdx.x;
    const float* recw_tile = lat.rec_w + (size_t)tpos.tile * SPLATS + threadIdx.x;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        l[r] = valid ? rec_tile[r * TP] : 0;
        w[r] = valid ? recw_tile[r * TP] : 0.f;
    }
    if (first) wait_for_previous_kernel();
    else __syncthreads();   // the rows before these have been read
    const float4* v4 = reinterpret_cast<const float4*>(v);
    stage_rows<PD, VP>(rows_s, nrows, lat.list_ref, info.x, v4);
    cp_async_wait_all();
    __syncthreads();
    float acc[VP];
    mix_rows_of_point<PD, VP>(acc, valid, l, w, rows_s, nrows, info.y, rows_cap, lat.list_ref, info.x, v4);
    const int last = C - (VP - 4);   // channels in the row's last quad; the next one is the homogeneous channel
    const float norm = last == 0 ? acc[VP - 4] : last == 1 ? acc[VP - 3] : last == 2 ? acc[VP - 2] : acc[VP - 1];
    const float inv = (float)(1.0 / (double)norm);
#pragma unroll
    for (int j = 0; j < VP; j++) {
        const float x = PL_FMUL(weight, PL_FMUL(acc[j], inv));
        m[j] = first ? x : PL_FADD(m[j], x);
    }
}
template <int PDA, int PDS, int VP, int CT>
__global__ void __launch_bounds__(Cfg<PDA>::TP, 3)
crf_slices(Geom g, float* __restrict__ q_out, const float* __restrict__ unaries, LatticeRows a, LatticeRows s,
           const float* __restrict__ va, const float* __restrict__ vs, float wa, float ws, int labels, int bulk_in, int bulk_out) {
    using CS = CrfSlices<PDA, PDS, VP>;
    constexpr int TP = CS::TP;
    const int C = CT ? CT : labels, US = CS::stride(C);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* rows_s = reinterpret_cast<float*>(smem_raw);                          // [ROWS][RS], then [TP][C]
    float* un_s = reinterpret_cast<float*>(smem_raw + CS::REGION);               // [TP][US]
    int* prow_s = reinterpret_cast<int*>(un_s + ((TP * US + 3) & ~3));           // [TP]
    __shared__ __align__(8) u64 bar;
    __shared__ u32 status_s;
    const int tid = threadIdx.x;
    const TilePos tpos = this_tile(g);
    int item, pix;
    const bool valid = tile_point(g, tpos, tid, item, pix);
    prow_s[tid] = valid ? item * g.n + pix : -1;
    if (tid == 0) {
        status_s = a.hdr->status | s.hdr->status;   // older than any blur pass, as all that is read before the wait
        if (bulk_in) mbar_init(&bar, 1);
    }
    const int nvalid = __syncthreads_count(valid);
    if (status_s != 0) {
        poison_tile_output(g, q_out, C);
        wait_for_previous_kernel();
        return;
    }
    if (bulk_in) {
        if (tid == 0) mbar_expect_tx(&bar, (unsigned)nvalid * C * 4u);
        if (tid < g.TY) {
            int row0, count;
            if (tile_row(g, tpos, tid, row0, count))
                bulk_load(un_s + (size_t)tid * g.TX * C, unaries + (size_t)row0 * C, (unsigned)count * C * 4u, &bar);
        }
    } else {
        const int DP = TP / C, DJ = TP - DP * C;   // element k = tid, tid + TP, ... is label j of point p
        int p = tid / C, j = tid - p * C;
        for (int it = 0; it < C; it++) {
            const int row = prow_s[p];
            if (row >= 0) cp_async4(un_s + p * US + j, unaries + (size_t)row * C + j);
            p += DP;
            j += DJ;
            if (j >= C) {
                j -= C;
                p++;
            }
        }
    }
    float m[VP];
    slice_message<PDA, VP>(m, wa, true, tpos, valid, a, va, rows_s, CS::ROWS, C);
    slice_message<PDS, VP>(m, ws, false, tpos, valid, s, vs, rows_s, CS::ROWS, C);
    const bool arrived = bulk_in ? mbar_wait(&bar, 0) : true;   // (else they came with the rows)
    if (!__syncthreads_and(arrived ? 1 : 0)) {   // every cached row has been read, too: the output may overwrite them
        if (tid == 0) atomicOr(&a.hdr->status, 1u << PL_INTERNAL_ERROR);
        mbar_wait(&bar, 0);
        poison_tile_output(g, q_out, C);
        return;
    }
    if (valid) {
        const float* u = un_s + tid * US;
        float sum = 0.f, mx = -INFINITY, den = 0.f;
#pragma unroll
        for (int j = 0; j < VP; j++)
            if (j < C) sum = PL_FADD(sum, m[j]);
#pragma unroll
        for (int j = 0; j < VP; j++)
            if (j < C) {
                m[j] = PL_FADD(-u[j], -PL_FADD(sum, -m[j]));
                mx = fmaxf(mx, m[j]);
            }
#pragma unroll
        for (int j = 0; j < VP; j++)
            if (j < C) {
                m[j] = expf(PL_FADD(m[j], -mx));
                den = PL_FADD(den, m[j]);
            }
        const float inv = PL_FDIV(1.f, den);
        float* o = rows_s + tid * C;
#pragma unroll
        for (int j = 0; j < VP; j++)
            if (j < C) o[j] = PL_FMUL(m[j], inv);
    }
    if (bulk_out) {
        fence_async_proxy();
        __syncthreads();
        if (tid < g.TY) {
            int row0, count;
            if (tile_row(g, tpos, tid, row0, count))
                bulk_store(q_out + (size_t)row0 * C, rows_s + (size_t)tid * g.TX * C, (unsigned)count * C * 4u);
            bulk_store_finish();
        }
    } else {
        __syncthreads();
        const int DP = TP / C, DJ = TP - DP * C;
        int p = tid / C, j = tid - p * C;
        for (int k = tid; k < TP * C; k += TP) {
            const int row = prow_s[p];
            if (row >= 0) q_out[(size_t)row * C + j] = rows_s[k];
            p += DP;
            j += DJ;
            if (j >= C) {
                j -= C;
                p++;
            }
        }
    }
}

}  // namespace pl
