// Small lattices: the index stage in one launch and all blur passes in one launch, each by a single cluster of
// CTAs that meets at the cluster's barrier between the phases.
//
// A call on a thumbnail is bound by its launches, on the host (2 us and more each) and on the device (a kernel with
// next to nothing to do takes about as long): three for the index, pd + 1 for the blur.  A cluster barrier costs less
// than a launch, and unlike a barrier over the whole grid it needs no cooperative launch and no memory to spin on.
// One cluster has the threads for lattices of up to SMALL_ENTRIES entries and SMALL_ITEMS 16-byte pieces of rows;
// beyond, the wide launches are used (their figures stand at small_index()).
#pragma once
#include "common.cuh"
#include "lattice_build.cuh"
#include "blur_slice.cuh"

namespace pl {

constexpr int SMALL_CTAS = 8, SMALL_THREADS = 1024;   // 8: the largest portable cluster

// All threads of the cluster; what any of them wrote before is visible to all after.
__device__ __forceinline__ void cluster_sync() {
    __threadfence();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// clear_table, insert_entries and link_neighbours.  What another CTA wrote in an earlier phase is read from L2.  A
// table slot names the entry that created it throughout: its key in list_keys is older than this launch.
template <int PD, int KW = Cfg<PD>::KW>
__global__ void __cluster_dims__(SMALL_CTAS, 1, 1) __launch_bounds__(SMALL_THREADS)
index_small(Header* hdr, u64* table, u32 max_log2, const Key<KW>* __restrict__ list_keys, u32* list_ref,
            u32* vid, Key<KW>* vkeys, VertexInit vi, Watch watch) {
    after_previous_kernel();
    const u32 tid = blockIdx.x * SMALL_THREADS + threadIdx.x, threads = SMALL_CTAS * SMALL_THREADS;
    if (call_failed(hdr)) {   // the same answer in every CTA: nothing sets the status before the first barrier
        report_to(watch, hdr);
        return;
    }
    const u32 T = hdr->num_entries;
    u32 lg = 10;
    while (lg < max_log2 && (1u << lg) < 2 * T) lg++;
    if (tid == 0) hdr->table_log2 = lg;
    const u32 mask = (1u << lg) - 1;
    for (u32 i = tid; i <= mask; i += threads) table[i] = EMPTY_SLOT;
    cluster_sync();

    int2* nb = reinterpret_cast<int2*>(vi.nbr);
    const int lane = threadIdx.x & 31;
    for (u32 t0 = tid - lane; t0 < T; t0 += threads) {   // a warp's entries; all its lanes make the same trips
        const u32 t = t0 + lane;
        bool winner = false;
        Key<KW> k;
        if (t < T) {
            k = list_keys[t];
            const u64 h = hash_key<KW>(k);
            const u64 mine = (h & 0xFFFFFFFF00000000ull) | (u64)t;
            u32 ref = 0xFFFFFFFFu, s = (u32)h & mask;
            for (u32 it = 0; it <= mask; it++) {
                u64 cur = __ldcg(&table[s]);
                if (cur == EMPTY_SLOT) {
                    cur = atomicCAS(&table[s], EMPTY_SLOT, mine);
                    if (cur == EMPTY_SLOT) {
                        ref = t;
                        winner = true;
                        break;
                    }
                }
                if ((u32)(cur >> 32) == (u32)(h >> 32) && key_equal<KW>(list_keys[(u32)cur], k)) {
                    ref = (u32)cur;
                    break;
                }
                s = (s + 1) & mask;
            }
            if (ref == 0xFFFFFFFFu) {
                atomicOr(&hdr->status, 1u << PL_INTERNAL_ERROR);
                ref = t;
                winner = true;
            }
            list_ref[t] = ref;
        }
        const unsigned won = __ballot_sync(0xFFFFFFFFu, winner);
        u32 first = 0;
        if (lane == 0 && won) first = atomicAdd(&hdr->num_vertices, (u32)__popc(won));
        first = __shfl_sync(0xFFFFFFFFu, first, 0);
        if (winner) {
            const u32 v = first + __popc(won & ((1u << lane) - 1u));
            vid[t] = v;
            vkeys[v] = k;
#pragma unroll
            for (int a = 0; a <= PD; a++) nb[(u64)a * vi.max_entries + v] = make_int2(-1, -1);
            if (vi.rows) {
                uint4* row = reinterpret_cast<uint4*>(static_cast<unsigned char*>(vi.rows) + (u64)v * vi.row_bytes);
                for (u32 i = 0; i < vi.row_bytes / 16; i++) row[i] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    }
    cluster_sync();

    if (tid == 0) report_to(watch, hdr);
    const u32 M = __ldcg(&hdr->num_vertices);
    for (u32 t = tid; t < T; t += threads) list_ref[t] = __ldcg(&vid[list_ref[t]]);   // the thread's own words
    for (u32 i = tid; i < M * (PD + 1); i += threads) {
        const u32 a = i / M, v = i - a * M;
        Key<KW> k = load_key_l2<KW>(&vkeys[v]);
#pragma unroll
        for (int j = 0; j < KW; j++) k.w[j] += axis_word<PD>((int)a, j);
        const u64 h = hash_key<KW>(k);
        u32 s = (u32)h & mask;
        for (u32 it = 0; it <= mask; it++) {
            const u64 cur = __ldcg(&table[s]);
            if (cur == EMPTY_SLOT) break;
            if ((u32)(cur >> 32) == (u32)(h >> 32) && key_equal<KW>(list_keys[(u32)cur], k)) {
                const u32 u = __ldcg(&vid[(u32)cur]);
                vi.nbr[2 * ((u64)a * vi.max_entries + v)] = (int)u;
                vi.nbr[2 * ((u64)a * vi.max_entries + u) + 1] = (int)v;
                break;
            }
            s = (s + 1) & mask;
        }
    }
}

// All blur passes (see blur_axis): from v0 to v1 and back, pass by pass.
template <typename V>
__global__ void __cluster_dims__(SMALL_CTAS, 1, 1) __launch_bounds__(SMALL_THREADS)
blur_small(const Header* hdr, const int* __restrict__ nbr, u64 max_entries, V* v0, V* v1, u32 vpr, int axes,
           int reverse) {
    const u32 tid = blockIdx.x * SMALL_THREADS + threadIdx.x, threads = SMALL_CTAS * SMALL_THREADS;
    const u32 M = hdr->num_vertices, items = M * vpr, v_first = tid / vpr;   // (older than the splat before this)
    const int2* __restrict__ nb = reinterpret_cast<const int2*>(nbr);
    auto axis = [&](int step) { return (u64)(reverse ? axes - 1 - step : step) * max_entries; };
    int2 ahead = tid < items ? __ldg(nb + axis(0) + v_first) : make_int2(-1, -1);   // neighbours of the first item
    after_previous_kernel();
    if (call_failed(hdr)) return;   // nothing sets the status from here on: the same answer in every CTA
    const V zero = {};
    V *src = v0, *dst = v1;
    for (int step = 0; step < axes; step++) {
        const int2* __restrict__ nb_axis = nb + axis(step);
        for (u32 e = tid; e < items; e += threads) {
            const u32 v = e / vpr, j = e - v * vpr;
            const int2 n = e == tid ? ahead : __ldg(nb_axis + v);
            const V b = __ldcg(src + e);
            const V a = n.x >= 0 ? __ldcg(src + (u32)n.x * vpr + j) : zero;
            const V c = n.y >= 0 ? __ldcg(src + (u32)n.y * vpr + j) : zero;
            dst[e] = mix_rows(a, b, c);
        }
        if (step + 1 < axes) {
            if (tid < items) ahead = __ldg(nb + axis(step + 1) + v_first);
            cluster_sync();
        }
        V* const t = src;
        src = dst;
        dst = t;
    }
}

}  // namespace pl
