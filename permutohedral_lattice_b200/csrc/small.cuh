// Small lattices: the index stage in one launch, and all blur passes in one launch of clusters whose shared memory holds
// the rows.
//
// A call on a thumbnail is bound by its launches, on the host (2 us and more each) and on the device (a kernel with
// next to nothing to do takes about as long): three for the index, pd + 1 for the blur, and inside each of them by round
// trips to L2 that depend on one another.  So here the table lies in shared memory, and so do the rows.
#pragma once
#include "common.cuh"
#include "lattice_build.cuh"
#include "blur_slice.cuh"

namespace pl {

constexpr int SMALL_THREADS = 1024;

// clear_table, insert_entries and link_neighbours.  Every CTA builds the whole table for itself, in shared memory, and
// then does its share of what goes to global memory: nothing is exchanged between CTAs, so there is no barrier over them,
// no atomic and no probe in L2.  They agree on the vertices because a key belongs to its first entry, whatever order the
// threads came in, and vertices are numbered in the order of those entries.  33x45 x 3, 3074 entries: 17.8 us by one cluster
// of eight CTAs on a table in global memory, 9.4 so, of it 2.5 in the compare-and-swaps (writing numbers and reading them
// back in rounds, as the tiles do, took 3.5).
//
// Shared memory of `bytes`, for T entries: the keys (pd up to 5: first_s [T] and, beyond pd 3, rest_s [T]; else their
// linear hashes [T], the key itself being compared in global memory), the slot of every entry [T], the entry of every
// vertex [T], the rest slots of 32 bits: vertex << 16 | entry.  A CTA's threads are few for its work, which is bound by
// their instructions: hence a hash of 32 bits, linear in the key like the global table's, and its upper part for the slot.
constexpr u32 SMALL_MAX_ENTRIES = 10240;   // numbers fit 16 bits, the table fits a block's shared memory
template <int PD>
struct SmallIndex {
    static constexpr bool EXACT = Cfg<PD>::KEY_SLOTS, REST = EXACT && Cfg<PD>::KW > 1;
    static constexpr u32 PER_ENTRY = 8 + (REST ? 4 : 0) + 2 + 2;
    __host__ __device__ static constexpr u32 fixed(u32 entries) { return ((entries + 7u) & ~7u) * PER_ENTRY; }
    // Four slots an entry, or as many as fit, 1.5 at least: a warp waits for the longest of its 32 walks.
    __host__ __device__ static constexpr size_t bytes(u32 entries) {
        const size_t most = 220 * 1024, whole = fixed(entries) + 16ull * entries + 256;
        return whole < most ? whole : most;
    }
    static_assert(fixed(SMALL_MAX_ENTRIES) + 6ull * SMALL_MAX_ENTRIES <= 222 * 1024, "1.5 slots an entry");
};

PL_CX u32 small_factor(int j) { return (u32)(hash_factor(j + 16) >> 32) | 1u; }
__device__ __forceinline__ u32 small_hash(u64 first) {
    return (u32)first * small_factor(0) + (u32)(first >> 32) * small_factor(1);
}

// SHARED: the lattice serves several items (see ItemRows).  A kernel of its own: with the loops over all items in it, it took 22.1 -> 23.0 us
// for 7000 entries of one lattice, and 9.9 -> 10.4 for 2800 (2x48x64 x 1 45.3 -> 47.1 a call).
template <int PD, int KW, bool SHARED>
__global__ void __launch_bounds__(SMALL_THREADS)
index_small(Header* hdr, const Key<KW>* __restrict__ list_keys, u32* __restrict__ list_ref,
            Key<KW>* __restrict__ vkeys, VertexInit vi, ItemRows rows, u32 smem_bytes, Watch watch) {
    after_previous_kernel();
    using SI = SmallIndex<PD>;
    constexpr int WARPS = SMALL_THREADS / 32, CHUNKS = SMALL_MAX_ENTRIES / SMALL_THREADS;
    constexpr u32 FREE = 0xFFFFFFFFu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ u32 warp_first[CHUNKS * WARPS], vertices_s;
    const uint4 counts = __ldcg(reinterpret_cast<const uint4*>(hdr));   // entries, vertices, status, table
    if (counts.z != 0) {   // final by now: the same in every thread
        report_to(watch, hdr);
        return;
    }
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 T = counts.x, TA = (T + 7u) & ~7u;   // (at most the bound that smem_bytes is for)
    u64* const first_s = reinterpret_cast<u64*>(smem_raw);                            // keys or hashes
    u32* const rest_s = reinterpret_cast<u32*>(first_s + TA);
    u16* const slot_s = reinterpret_cast<u16*>(rest_s + (SI::REST ? TA : 0));         // entry -> slot
    u16* const owner_s = slot_s + TA;                                                 // vertex -> entry
    u32* const table_s = reinterpret_cast<u32*>(owner_s + TA);
    const u32 slots = min((smem_bytes - SI::fixed(T)) / 4u, max(4u * T, 64u));
    constexpr u32 AHEAD = KW <= 2 ? 4 : 2;   // keys in flight
    for (u32 t0 = tid; t0 < T; t0 += AHEAD * SMALL_THREADS) {
        Key<KW> k[AHEAD];
#pragma unroll
        for (u32 c = 0; c < AHEAD; c++) k[c] = list_keys[min(t0 + c * SMALL_THREADS, T - 1)];
#pragma unroll
        for (u32 c = 0; c < AHEAD; c++) {
            const u32 t = t0 + c * SMALL_THREADS;
            if (t < T) {
                first_s[t] = SI::EXACT ? k[c].w[0] : linear_hash<KW>(k[c]);
                if constexpr (SI::REST) rest_s[t] = (u32)k[c].w[KW - 1];
            }
        }
    }
    for (u32 i = tid; i < slots; i += SMALL_THREADS) table_s[i] = FREE;
    __syncthreads();

    auto hash = [&](u32 t) -> u32 {   // of entry t's key
        u32 h = small_hash(first_s[t]);
        if constexpr (SI::REST) h += rest_s[t] * small_factor(2);
        return h;
    };
    auto slot_of = [&](u32 h) -> u32 { return __umulhi(h, slots); };

    for (u32 t = tid; t < T; t += SMALL_THREADS) {
        u32 s = slot_of(hash(t));
        for (u32 it = 0; it < slots; it++) {
            u32 cur = *reinterpret_cast<volatile u32*>(table_s + s);
            if (cur == FREE) {
                cur = atomicCAS(table_s + s, FREE, t);
                if (cur == FREE) break;
            }
            bool same = first_s[cur] == first_s[t];
            if constexpr (SI::REST) same = same && rest_s[cur] == rest_s[t];
            if constexpr (!SI::EXACT) same = same && key_equal<KW>(list_keys[cur], list_keys[t]);
            if (same) {
                if (t < cur) atomicMin(table_s + s, t);
                break;
            }
            s = s + 1 < slots ? s + 1 : 0;
        }
        slot_s[t] = (u16)s;
    }
    __syncthreads();

    // vertex numbers: the entries that stand in their slot, counted warp by warp
    u32 mine = 0;   // bit c: the entry tid + c SMALL_THREADS does
#pragma unroll
    for (int c = 0; c < CHUNKS; c++) {
        if (c * SMALL_THREADS < T) {
            const u32 t = c * SMALL_THREADS + tid;
            const bool owner = t < T && table_s[slot_s[t]] == t;
            const u32 all = __ballot_sync(0xFFFFFFFFu, owner);
            if (lane == 0) warp_first[c * WARPS + warp] = __popc(all);
            if (owner) mine |= 1u << c;
        }
    }
    __syncthreads();
    if (warp == 0) {
        u32 before = 0;
        for (u32 c = 0; c * SMALL_THREADS < T; c++) {
            const u32 n = warp_first[c * WARPS + lane];
            u32 incl = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u32 up = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if ((int)lane >= d) incl += up;
            }
            warp_first[c * WARPS + lane] = before + incl - n;
            before += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        if (lane == 0) vertices_s = before;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CHUNKS; c++) {
        if (c * SMALL_THREADS < T) {
            const bool owner = (mine >> c) & 1u;
            const u32 all = __ballot_sync(0xFFFFFFFFu, owner);
            if (owner) {
                const u32 t = c * SMALL_THREADS + tid, v = warp_first[c * WARPS + warp] + __popc(all & ((1u << lane) - 1u));
                owner_s[v] = (u16)t;
                table_s[slot_s[t]] = v << 16 | t;
            }
        }
    }
    __syncthreads();

    // this CTA's share
    const u32 M = vertices_s, me = blockIdx.x * SMALL_THREADS + tid, all = gridDim.x * SMALL_THREADS;
    if (me == 0) {
        hdr->num_vertices = M;
        u32 lg = 0;
        while ((1u << lg) < slots) lg++;
        hdr->table_log2 = lg;
        report_to(watch, hdr);
    }
    for (u32 t = me; t < T; t += all) {
        const u32 v = table_s[slot_s[t]] >> 16;
        if constexpr (!SHARED) list_ref[t] = v;
        if (owner_s[v] == t) {
            if constexpr (SI::EXACT) {
                Key<KW> k;
                k.w[0] = first_s[t];
                if constexpr (SI::REST) k.w[KW - 1] = rest_s[t];
                vkeys[v] = k;
            } else {
                vkeys[v] = list_keys[t];
            }
        }
    }
    if constexpr (SHARED) {
        for_entries_of(rows, T, me, all, [&](u32 t) { return table_s[slot_s[t]] >> 16; },
                       [&](u32 t, u32 b, u32 v) { store_vertex_of(rows, list_ref, t, b, v); });
        zero_rows_of(rows, M, me, all);
    } else if (rows.rows) {   // (fewer than 2^32 pieces)
        for (u32 i = me; i < M * rows.row_quads; i += all) rows.rows[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    int2* nb = reinterpret_cast<int2*>(vi.nbr);
    for (u32 i = me; i < M * (PD + 1); i += all) {
        const u32 a = i / M, v = i - a * M, t = owner_s[v];
        // what moving along axis a adds to the key and to its linear hash
        u64 move[KW], move_lin = 0;
#pragma unroll
        for (int j = 0; j < KW; j++) {
            move[j] = axis_word<PD>((int)a, j);
            move_lin += move[j] * hash_factor(j);
        }
        int found[2];
#pragma unroll
        for (int way = 0; way < 2; way++) {   // the "+" and the "-" neighbour (see link_neighbours)
            const u64 want = first_s[t] + (SI::EXACT ? (way ? 0ull - move[0] : move[0]) : way ? 0ull - move_lin : move_lin);
            u32 want_rest = 0;
            if constexpr (SI::REST) want_rest = rest_s[t] + (u32)(way ? 0ull - move[KW - 1] : move[KW - 1]);
            u32 s = slot_of(small_hash(want) + (SI::REST ? want_rest * small_factor(2) : 0u));
            found[way] = -1;
            for (u32 it = 0; it < slots; it++) {
                const u32 cur = table_s[s];
                if (cur == FREE) break;
                const u32 e = cur & 0xFFFFu;
                bool same = first_s[e] == want;
                if constexpr (SI::REST) same = same && rest_s[e] == want_rest;
                if constexpr (!SI::EXACT) {
                    if (same) {
                        Key<KW> k = list_keys[t];
#pragma unroll
                        for (int j = 0; j < KW; j++) k.w[j] += way ? 0ull - move[j] : move[j];
                        same = key_equal<KW>(list_keys[e], k);
                    }
                }
                if (same) {
                    found[way] = (int)(cur >> 16);
                    break;
                }
                s = s + 1 < slots ? s + 1 : 0;
            }
        }
        nb[(u64)a * vi.max_entries + v] = make_int2(found[0], found[1]);
    }
}

// All blur passes (see blur_axis) in one launch: channels never meet, so a cluster takes 16 bytes of every row (V: float4 or
// double2) and keeps them in its shared memory, twice (a pass reads one copy, of any CTA, and writes the other).  Each CTA has
// a run of 2^chunk_log2 vertices, at most PIECES a thread; between passes the cluster's barrier.  The rows come from v
// and go back there.  33x45 x 3, 2640 vertices, six passes: by one cluster through global memory, with the round trip to L2 and a
// fence besides the barrier in every pass, 12.7 us, so 7.
constexpr int SMALL_CTAS = 8;   // the largest portable cluster
// Not the .aligned form: between the branches around it the compiler need not bring a warp's threads together, and that
// form is an illegal instruction then.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float4 load_cluster(u32 addr, u32 cta, float4) {
    float4 x;
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                 : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                 : "r"(addr), "r"(cta)
                 : "memory");
    return x;
}
__device__ __forceinline__ double2 load_cluster(u32 addr, u32 cta, double2) {
    double2 x;
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %2, %3;\n\tld.shared::cluster.v2.f64 {%0, %1}, [a];\n\t}"
                 : "=d"(x.x), "=d"(x.y)
                 : "r"(addr), "r"(cta)
                 : "memory");
    return x;
}
template <typename V, int PIECES>
__global__ void __cluster_dims__(SMALL_CTAS, 1, 1) __launch_bounds__(SMALL_THREADS)
blur_small(const Header* hdr, const int* __restrict__ nbr, u64 max_entries, V* v, u32 vpr, int axes, int reverse) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* const buf = reinterpret_cast<V*>(smem_raw);
    const u32 M = hdr->num_vertices;   // (older than the splat before this)
    u32 chunk_log2 = 5;
    while ((u32)SMALL_CTAS << chunk_log2 < M) chunk_log2++;
    const u32 chunk = 1u << chunk_log2, first = (blockIdx.x % SMALL_CTAS) << chunk_log2;
    v += blockIdx.x / SMALL_CTAS;
    const int2* __restrict__ nb = reinterpret_cast<const int2*>(nbr);
    auto axis = [&](int step) { return (u64)(reverse ? axes - 1 - step : step) * max_entries; };
    int2 even[PIECES], odd[PIECES];   // neighbours of vertex first + at(p) in the next pass of either kind
    V mid[PIECES];
    auto at = [&](int p) { return threadIdx.x + p * SMALL_THREADS; };
    auto there = [&](int p) { return at(p) < chunk && first + at(p) < M; };
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
        if (there(p)) {
            even[p] = __ldg(nb + axis(0) + first + at(p));
            odd[p] = __ldg(nb + axis(1) + first + at(p));
        }
    }
    after_previous_kernel();
    if (call_failed(hdr)) return;   // nothing sets the status from here on: the same answer in every CTA
#pragma unroll
    for (int p = 0; p < PIECES; p++)
        if (there(p)) buf[at(p)] = mid[p] = __ldcg(v + (u64)(first + at(p)) * vpr);
    cluster_sync();
    const u32 base = (u32)__cvta_generic_to_shared(buf);
    const V zero = {};
    auto pass = [&](int step, int2 (&n)[PIECES], u32 from, u32 to) {   // from, to: the copies' first pieces
        auto row = [&](int u) {
            return u < 0 ? zero : load_cluster(base + (from + ((u32)u & (chunk - 1u))) * 16u, (u32)u >> chunk_log2, zero);
        };
#pragma unroll
        for (int p = 0; p < PIECES; p++) {
            if (there(p)) {
                mid[p] = mix_rows(row(n[p].x), mid[p], row(n[p].y));
                // two passes ahead, so that no pass waits for a round trip to L2
                if (step + 2 < axes) n[p] = __ldg(nb + axis(step + 2) + first + at(p));
                if (step + 1 < axes) buf[to + at(p)] = mid[p];
                else v[(u64)(first + at(p)) * vpr] = mid[p];
            }
        }
        cluster_sync();   // after the last pass too: no CTA leaves while another reads its rows
    };
    for (int step = 0; step < axes; step += 2) {
        pass(step, even, 0u, chunk);
        if (step + 1 < axes) pass(step + 1, odd, chunk, 0u);
    }
}

}  // namespace pl
