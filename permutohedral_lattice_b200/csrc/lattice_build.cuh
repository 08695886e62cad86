// Lattice construction: per-tile key generation and de-duplication (build_tiles), the global hash
// table (clear_table, insert_entries) and the vertex / neighbour tables (insert_entries, link_neighbours).
#pragma once
#include <type_traits>
#include "common.cuh"

namespace pl {

// The header and the sketch before a call.  A kernel and not a memset, so that build_tiles can start beside it (the gap between a memset and the
// build, 3 to 4 us a call: 8 x 512x512 x 21, pd 2, forward + backward, 431 -> 425; 512x512 x 3 in double 188.5 -> 185.5).  The host needs a
// microsecond more for it.
// It also clears (to ones: empty slots) what the index stage needs, the direct index or the whole table that the call's bound allows,
// where that is at most 16 MB, so that no launch between the build and the insert has to, and the call keeps no sketch: us a call, 2 x
// 48x64 x 3 52 / 46, 4 x 180x240 x 3 60 / 57, 60x70 x 2 without a guide 32 / 28, five CRF steps on
// 375x500 x 21 with both builds 413 / 405, 512x512 x 3 in double, forward + backward, 175 / 167.  At 32 MB nothing is left of it (2 x 512x512 x 21,
// deterministic, 407 / 406).  (By build_tiles, a share a tile, it cost calls without any
// 0.7 %.)
struct ClearTable {
    uint4* table;   // null: a launch of its own does
    u32 quads;      // 16 bytes each
};
constexpr u32 CLEAR_QUADS = 1u << 20;         // 16 MB, at most; 8 MB where the build waits for it at its start (pd 16)
constexpr u32 CLEAR_QUADS_ALONE = 1u << 19;
__global__ void __launch_bounds__(256) clear_header(Header* hdr, u32 quads, ClearTable clear) {
    after_previous_kernel();
    if (blockIdx.x == 0)
        for (u32 i = threadIdx.x; i < quads; i += 256) reinterpret_cast<uint4*>(hdr)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (u32 i = blockIdx.x * 256 + threadIdx.x; i < clear.quads; i += gridDim.x * 256)
        clear.table[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
}

// ---------------------------------------------------------------------------------------------
// build_tiles
// ---------------------------------------------------------------------------------------------
// R: number type of the call (float or double); it decides the geometry arithmetic and the type of the
// stored weights, nothing else.
template <typename R>
struct is_double { static constexpr bool value = false; };
template <>
struct is_double<double> { static constexpr bool value = true; };

// x << s with 0 for every shift beyond the word (negative ones included).
__device__ __forceinline__ u32 shift_in(u32 x, u32 s) {
    u32 y;
    asm("shl.b32 %0, %1, %2;" : "=r"(y) : "r"(x), "r"(s));
    return y;
}

// The keys of one point, remainder by remainder (src/PermutohedralLatticeCPU.h:297-304): coordinate i of the
// remainder-r vertex is rem0_i + r - (PD+1) [rank_i > PD - r], so a step from r - 1 to r adds one to every
// coordinate and takes PD+1 off the one of rank PD - r + 1.  Coordinates are packed two to a word, biased by
// 0x8000 (no carries between them); `perm` holds the coordinate of every rank >= 1 in four bits.
template <int PD>
struct PointKeys {
    static constexpr int CW = Cfg<PD>::CW;
    static constexpr bool WIDE = PD > 8;
    u32 w[CW];
    u32 perm, perm_hi;   // coordinates of ranks 1..8 and 9..16
    int last_rank;       // WIDE: rank of coordinate PD, which is not stored (else its nibble is 15: no coordinate)

    template <typename S>
    __device__ __forceinline__ void start(const S& s) {
#pragma unroll
        for (int j = 0; j < CW; j++) {
            const u32 lo = rem0_low16<PD>(s, 2 * j);
            w[j] = (2 * j + 1 < PD) ? __byte_perm(lo, rem0_low16<PD>(s, 2 * j + 1 < PD ? 2 * j + 1 : 0), 0x5410) ^ 0x80008000u
                                    : (lo & 0xFFFFu) ^ 0x8000u;
        }
        perm = perm_hi = 0;
#pragma unroll
        for (int i = 1; i < PD; i++) {
            perm += shift_in((u32)i, (u32)(4 * s.rank[i] - 4));
            if constexpr (WIDE) perm_hi += shift_in((u32)i, (u32)(4 * s.rank[i] - 36));
        }
        if constexpr (!WIDE) perm += shift_in(15u, (u32)(4 * s.rank[PD] - 4));
        last_rank = s.rank[PD];
    }
    __device__ __forceinline__ u32 moved16(int r) const {   // 16 x the coordinate that a step to r takes a cell off
        const int rank = PD - r + 1;
        if constexpr (WIDE) {
            const u32 c16 = ((rank > 8 ? perm_hi >> (4 * (rank - 9)) : perm >> (4 * (rank - 1))) & 15u) * 16u;
            return rank == last_rank ? 512u : c16;
        } else {
            return ((rank > 1) ? perm >> (4 * (rank - 2)) : perm << 4) & 0xF0u;
        }
    }
    __device__ __forceinline__ u32 moves(u32 c16, int j) const {   // what that step adds to word j
        return ((2 * j + 1 < PD) ? 0x00010001u : 1u) - shift_in((u32)(PD + 1), c16 - 32u * j);
    }
    // from remainder r - 1 to remainder r, and back
    __device__ __forceinline__ void step(int r) {
        const u32 c16 = moved16(r);
#pragma unroll
        for (int j = 0; j < CW; j++) w[j] += moves(c16, j);
    }
    __device__ __forceinline__ void step_back(int r) {
        const u32 c16 = moved16(r);
#pragma unroll
        for (int j = 0; j < CW; j++) w[j] -= moves(c16, j);
    }
    // 32-bit hash of the key (of item `seed`): its high bits place the key in the tile's table
    __device__ __forceinline__ u32 hash(u32 seed) const {
        u32 h = seed;
#pragma unroll
        for (int j = 0; j < CW; j++) h += w[j] * (u32)(hash_factor(j + 8) >> 32 | 1u);
        return h;
    }
};

// What the tile keeps of its points' keys in shared memory.  Up to pd = 8: the coordinate words of every splat's
// key.  Above (COMPACT): per point the remainder-0 key and the ranks of its coordinates, one byte each, from
// which the key of any remainder follows.
template <int PD>
struct TileKeys {
    static constexpr int TP = Cfg<PD>::TP, CW = Cfg<PD>::CW, KS = Cfg<PD>::KEY_WORDS;
    static constexpr bool COMPACT = Cfg<PD>::COMPACT;
    u32* s;
    // coordinate words of splat `id` = r * TP + point
    __device__ __forceinline__ void load(int id, int r, u32 (&k)[CW]) const {
        if constexpr (COMPACT) {
            const uint4* rec = reinterpret_cast<const uint4*>(s + (id - r * TP) * KS);
            u32 rank[4];
            const uint4 v = rec[CW / 4];
            rank[0] = v.x; rank[1] = v.y; rank[2] = v.z; rank[3] = v.w;
            const u32 above = (u32)(127 - (PD - r)) * 0x01010101u;   // rank + this has its top bit set iff rank > PD - r
#pragma unroll
            for (int j = 0; j < CW; j += 4) {
                const uint4 q = rec[j / 4];
                k[j] = q.x; k[j + 1] = q.y; k[j + 2] = q.z; k[j + 3] = q.w;
            }
#pragma unroll
            for (int j = 0; j < CW; j++) {
                const u32 taken = ((rank[j / 2] + above) >> 7) & 0x01010101u;
                const u32 fields = __byte_perm(taken, 0u, (j & 1) ? 0x4342 : 0x4140);   // two 16-bit fields
                k[j] += (u32)r * 0x00010001u - fields * (u32)(PD + 1);
            }
        } else if constexpr (KS == 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(s + id * 4);
            const u32 t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < CW; j++) k[j] = t[j];
        } else if constexpr (KS == 2) {
            const uint2 v = *reinterpret_cast<const uint2*>(s + id * 2);
            k[0] = v.x;
            k[CW - 1] = v.y;
        } else {
            k[0] = s[id];
        }
    }
    __device__ __forceinline__ void store(int id, const u32 (&k)[CW]) const {
        if constexpr (KS == 4)
            *reinterpret_cast<uint4*>(s + id * 4) = make_uint4(k[0], k[1 % CW], k[2 % CW], CW > 3 ? k[3 % CW] : 0u);
        else if constexpr (KS == 2)
            *reinterpret_cast<uint2*>(s + id * 2) = make_uint2(k[0], k[CW - 1]);
        else
            s[id] = k[0];
    }
    // is splat a, of any remainder, one of splat b's remainder r with b's key
    __device__ __forceinline__ bool same(int a, int b, int r) const {
        u32 diff = (u32)(a ^ b) & ~(u32)(TP - 1);
        if (COMPACT && diff) return false;   // a record is read by point and remainder
        u32 x[CW], y[CW];
        load(a, r, x);
        load(b, r, y);
#pragma unroll
        for (int j = 0; j < CW; j++) diff |= x[j] ^ y[j];
        return diff == 0;
    }
    // the same for a splat b whose key the caller holds (COMPACT)
    __device__ __forceinline__ bool same_as(int a, int b, int r, const u32 (&y)[CW]) const {
        if ((u32)(a ^ b) & ~(u32)(TP - 1)) return false;
        u32 x[CW], diff = 0;
        load(a, r, x);
#pragma unroll
        for (int j = 0; j < CW; j++) diff |= x[j] ^ y[j];
        return diff == 0;
    }
    __device__ __forceinline__ u32 hash(int id, int r, u32 seed) const {
        u32 k[CW];
        load(id, r, k);
        return hash(k, seed);
    }
    __device__ static __forceinline__ u32 hash(const u32 (&k)[CW], u32 seed) {
        u32 h = seed;
#pragma unroll
        for (int j = 0; j < CW; j++) h += k[j] * (u32)(hash_factor(j + 8) >> 32 | 1u);
        return h;
    }
    // the key as the global list holds it
    template <int KW>
    __device__ static __forceinline__ Key<KW> global_key(const u32 (&k)[CW], int item) {
        Key<KW> out;
#pragma unroll
        for (int j = 0; j < KW; j++) {
            const u32 lo = (2 * j < CW) ? k[2 * j < CW ? 2 * j : 0] : 0u;
            const u32 hi = (2 * j + 1 < CW) ? k[2 * j + 1 < CW ? 2 * j + 1 : 0] : 0u;
            out.w[j] = (u64)lo | ((u64)hi << 32);
        }
        if constexpr (KW * 4 > PD) key_set<KW>(out, PD, (u16)item);
        return out;
    }
};

// Sets the bit of a key, of tile hash h, in the sketch if the key is sampled (sketch_shift < 0: no sketch).
__device__ __forceinline__ void add_to_sketch(Header* hdr, u32 h, int sketch_shift) {
    if (sketch_shift < 0) return;
    const u32 x = (h ^ (h >> 15)) * 0x9E3779B1u;
    if ((x >> 1) < (0x80000000u >> sketch_shift)) {
        const u32 bit = (h ^ (x << 7)) * 0x85EBCA77u >> (32 - SKETCH_LOG2);
        atomicOr(reinterpret_cast<u32*>(hdr + 1) + (bit >> 5), 1u << (bit & 31u));
    }
}

constexpr u32 TILE_SEED = 0x2C1B3C6Du;    // times the item: keys of different items sample independently
constexpr int TILE_ROUNDS = 8;            // of the tile's de-duplication

// One thread per point of the tile: features, enclosing simplex, weights, keys; then the tile's keys are
// de-duplicated, its distinct keys appended to the global entry list, and every splat's entry number stored.
//
// De-duplication without atomics, in rounds: every splat writes its number into the slot of its key's hash (one
// of the writers stays), and after a barrier reads the slot back.  If the number there is of the same key, that
// splat represents the key, for all its splats alike, since all of them read that slot.  Keys that lost their slot
// to another key go into the next round with another hash; with 2.5 slots a splat that leaves a few per cent of
// them.  A splat still without representative after TILE_ROUNDS represents itself: the key then has two entries,
// which the global table merges as it does those of different tiles.  A splat stands only for splats of its own
// remainder, because entries are numbered remainder by remainder.  Keys of two remainders differ (a key modulo PD+1 is
// its remainder), but only until 16 bits, or the integers of a float, no longer hold their coordinates.
// (One compare-and-swap per splat on the slot, as before, took a third of the kernel's shared-memory wavefronts, and
// its retries most of the divergence.)
//
// Bound by issue slots and the LSU pipe.  Up to pd = 5 six CTAs fit an SM: the registers are capped at 40 for it
// (measured 13 % faster than five CTAs with 48).
// SORTED (float calls that build a lattice for reuse): also leave every tile's splats sorted by entry in
// `srec`, in the form the splat kernels walk, so that no later splat through this lattice sorts again.
// It costs this kernel a quarter more time and saves every splat a fifth: worth it from the second
// splat on, which is why the one-call filter does not ask for it.
// sketch_shift < 0: no sketch of the lattice's size (see SKETCH_LOG2).
// KW: words of a key (see Cfg).
template <int PD, typename R = float, bool SORTED = false, int KW = Cfg<PD>::KW>
__global__ void __launch_bounds__(Cfg<PD>::TP, (PD <= 5 && !is_double<R>::value) ? 6 : (Cfg<PD>::COMPACT && !is_double<R>::value) ? 5 : 1)
build_tiles(Geom g, const R* __restrict__ positions, const R* __restrict__ reference,
            Header* hdr, int2* __restrict__ tile_info, u16* __restrict__ rec, R* __restrict__ rec_w,
            uint2* __restrict__ srec, Key<KW>* __restrict__ list_keys, u32 max_entries, int sketch_shift) {
    // Launched to overlap clear_header, which starts when all before it has finished: only the header has to wait.
    if constexpr (Cfg<PD>::COMPACT) wait_for_previous_kernel();   // (whose sketch is kept from the start)
    constexpr int TP = Cfg<PD>::TP, SPLATS = Cfg<PD>::SPLATS, LSLOG = Cfg<PD>::LSLOG;
    constexpr bool COMPACT = Cfg<PD>::COMPACT;
    constexpr int KEYS = (int)Cfg<PD>::build_keys(SORTED);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileKeys<PD> keys;
    keys.s = reinterpret_cast<u32*>(smem_raw);
    u16* slots_s = reinterpret_cast<u16*>(smem_raw + KEYS);                       // [LS]
    u16* lidx_s = slots_s + Cfg<PD>::LS;                                          // [SPLATS]
    u16* rep_s = lidx_s + SPLATS;                                                 // [SPLATS], COMPACT only
    __shared__ int cnt_s[PD + 1], base_s;   // entries per remainder; first global entry of the tile
    __shared__ int wsum_s[TP / 32];
    __shared__ int open_s;   // COMPACT: splats without representative

    const TilePos tpos = this_tile(g);
    const int tid = threadIdx.x, tile = tpos.tile;
    if (tid <= PD) cnt_s[tid] = 0;
    if (COMPACT && tid == 0) open_s = 0;
    int item, pix, po, py, px;
    const bool valid = tile_point(g, tpos, tid, item, pix, po, py, px);
    u32 slot2[PD / 2 + 1];   // slots of the splats' keys, two to a word
#pragma unroll
    for (int r = 0; r <= PD / 2; r++) slot2[r] = 0;
    PointKeys<PD> k;
    if (valid) {
        R f[PD];
        R w[PD + 1];
        load_features<PD>(g, positions, reference, item, pix, po, py, px, f);
        typename std::conditional<is_double<R>::value, Simplex64<PD>, Simplex<PD>>::type s;
        if constexpr (is_double<R>::value) {
            find_simplex_f64<PD>(f, g.scale_d, s);
            barycentric_f64<PD>(s, w);
        } else {
            find_simplex<PD>(f, g.scale, s);
            barycentric<PD>(s, w);
        }
        // the weights are final: store them now so the writes overlap the de-duplication below
        R* recw_tile = rec_w + (size_t)tile * SPLATS;
#pragma unroll
        for (int r = 0; r <= PD; r++) store_once(recw_tile + r * TP + tid, w[r]);
        // COMPACT: a point's own key is formed by steps, that of a splat it is compared with from the stored ranks.
        // The two are the same once the ranks are a permutation.
        if constexpr (COMPACT) settle_ranks<PD>(s);
        k.start(s);
        if constexpr (COMPACT) {
            u32* mine = keys.s + tid * Cfg<PD>::KEY_WORDS;
#pragma unroll
            for (int j = 0; j < Cfg<PD>::CW; j++) mine[j] = k.w[j];
#pragma unroll
            for (int j = 0; j < 4; j++)
                mine[Cfg<PD>::CW + j] = (u32)s.rank[4 * j] | ((u32)s.rank[4 * j + 1] << 8) |
                                        ((u32)s.rank[4 * j + 2] << 16) | ((u32)s.rank[4 * j + 3] << 24);
        }
        const u32 seed = (u32)item * TILE_SEED;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            if (r > 0) k.step(r);
            if constexpr (!COMPACT) keys.store(r * TP + tid, k.w);
            const u32 h = k.hash(seed);
            const u32 slot = h >> (32 - LSLOG);
            slots_s[slot] = (u16)(r * TP + tid);
            if constexpr (COMPACT) lidx_s[r * TP + tid] = (u16)slot;   // (there are no entry numbers yet)
            else slot2[r / 2] |= slot << (16 * (r & 1));
            if constexpr (COMPACT) add_to_sketch(hdr, h, sketch_shift);   // (else once an entry, below)
        }
    }
    __syncthreads();

    int rep[COMPACT ? 1 : PD + 1];   // the splat that represents each splat's key (COMPACT: in rep_s)
    u32 open = 0;                    // splats without a representative
    auto set_rep = [&](int r, int v) {
        if constexpr (COMPACT) rep_s[r * TP + tid] = (u16)v;
        else rep[r] = v;
    };
    auto get_rep = [&](int r) -> int {
        if constexpr (COMPACT) return (int)rep_s[r * TP + tid];
        else return rep[r];
    };
    if constexpr (COMPACT) {
#pragma unroll 1
        for (int r = PD; r >= 0; r--) {   // the key is that of remainder PD by now and goes back step by step
            const int me = r * TP + tid;
            int c = me;
            if (valid) {
                c = slots_s[lidx_s[me]];
                if (c != me && !keys.same_as(c, me, r, k.w)) {
                    c = me;
                    open |= 1u << r;
                }
                if (r > 0) k.step_back(r);
            }
            set_rep(r, c);
        }
    } else {
#pragma unroll
        for (int r = 0; r <= PD; r++)
            rep[r] = valid ? (int)slots_s[(slot2[r / 2] >> (16 * (r & 1))) & 0xFFFFu] : r * TP + tid;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int me = r * TP + tid;
            if (rep[r] != me && !keys.same(rep[r], me, r)) {
                rep[r] = me;
                open |= 1u << r;
            }
        }
    }
    auto next_slot = [&](int id, int r, int round) {
        const u32 h = keys.hash(id, r, (u32)item * TILE_SEED) + (u32)round * 0x632BE5ABu;
        return ((h ^ (h >> 13)) * 0x85EBCA77u) >> (32 - LSLOG);
    };
    if constexpr (COMPACT) {
        // The open splats, a few in a hundred, are put in a list and the rounds run over that.  Looked for among all 17
        // splats of a point, most warps had one or another of every remainder and went through hash and comparison
        // for each: with it and the keys by steps 350 -> 286 us on 1 M points.  (With six splats a point, whose keys lie
        // in shared memory as they are, the list and its barriers cost more than they saved: 160 -> 170 us on 16 x
        // 512x512, pd 5.)
        u16* const list = lidx_s;
        __syncthreads();   // the slots kept there have been read
        if (open) {
            int pos = atomicAdd(&open_s, __popc(open));
            for (u32 rest = open; rest; rest &= rest - 1) list[pos++] = (u16)((__ffs(rest) - 1) * TP + tid);
        }
        __syncthreads();
        const int listed = open_s;
        u32 todo = 0;   // of the list's splats number tid + m TP, those still open
        for (int m = 0; tid + m * TP < listed; m++) todo |= 1u << m;
        for (int round = 1; listed && round <= TILE_ROUNDS; round++) {
            for (u32 rest = todo; rest; rest &= rest - 1) {
                const int id = list[tid + (__ffs(rest) - 1) * TP];
                slots_s[next_slot(id, id / TP, round)] = (u16)id;
            }
            __syncthreads();
            for (u32 rest = todo; rest; rest &= rest - 1) {
                const int m = __ffs(rest) - 1, id = list[tid + m * TP], c = slots_s[next_slot(id, id / TP, round)];
                if (c == id || keys.same(c, id, id / TP)) {
                    rep_s[id] = (u16)c;
                    todo &= ~(1u << m);
                }
            }
            if (!__syncthreads_or((int)todo)) break;
        }
    } else {
        for (int round = 1;; round++) {   // (left behind the barrier, when nobody reads a slot any more)
            if (!__syncthreads_or((int)open) || round > TILE_ROUNDS) break;
            if (open) {
#pragma unroll
                for (int r = 0; r <= PD; r++)
                    if ((open >> r) & 1u) slots_s[next_slot(r * TP + tid, r, round)] = (u16)(r * TP + tid);
            }
            __syncthreads();
            if (open) {
#pragma unroll
                for (int r = 0; r <= PD; r++) {
                    if ((open >> r) & 1u) {
                        const int me = r * TP + tid, c = slots_s[next_slot(me, r, round)];
                        if (c == me || keys.same(c, me, r)) {
                            rep[r] = c;
                            open &= ~(1u << r);
                        }
                    }
                }
            }
        }
    }
    // Number the tile's entries remainder by remainder (all entries of remainder 0 first, ...: the splat
    // stage, which walks the tile's splats in entry order, measured 4 % faster with this order than with
    // entries grouped by warp).  Per warp ONE shared-memory atomic instruction: lane r adds the warp's
    // number of new remainder-r entries to counter r.  The index stored now is relative to the
    // remainder's segment; the segment starts are known after the barrier.
    unsigned char* owner_s = reinterpret_cast<unsigned char*>(slots_s) + 4 * SPLATS;   // [SPLATS], in the dead hash too: see below
    int* run_s = reinterpret_cast<int*>(slots_s);   // SORTED: the tile hash is dead, its memory counts the splats of every entry
    if constexpr (SORTED) {
        static_assert(sizeof(int) * SPLATS <= sizeof(u16) * Cfg<PD>::LS, "the counters fit the hash's memory");
        __syncthreads();
        for (int i = tid; i < SPLATS; i += TP) run_s[i] = 0;
    }
    {
        const int lane = tid & 31;
        unsigned owners[PD + 1];
        unsigned mine = 0;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            owners[r] = __ballot_sync(0xFFFFFFFFu, valid && get_rep(r) == r * TP + tid);
            mine = (lane == r) ? owners[r] : mine;
        }
        int first = 0;
        if (lane <= PD && mine) first = atomicAdd(&cnt_s[lane], __popc(mine));
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int first_r = __shfl_sync(0xFFFFFFFFu, first, r);
            if ((owners[r] >> lane) & 1u) {
                const int at = first_r + __popc(owners[r] & ((1u << lane) - 1u));
                lidx_s[r * TP + tid] = (u16)at;
                if constexpr (!COMPACT) owner_s[r * TP + at] = (unsigned char)tid;
            }
        }
    }
    __syncthreads();
    int seg[PD + 1];   // first entry of each remainder's segment
    int cnt = 0;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        seg[r] = cnt;
        cnt += cnt_s[r];
    }
    wait_for_previous_kernel();
    if (tile == 0 && tid == 0) {
        hdr->capacity = g.lattice_items > 1 ? g.bound : max_entries;
        hdr->sorted = SORTED ? 1u : 0u;
        hdr->calm_entries = (u32)g.calm_entries;
        hdr->items = (u32)g.lattice_items;
        hdr->row_step = g.row_step;
    }
    if (tid == 0) {
        u32 base = atomicAdd(&hdr->num_entries, (u32)cnt);
        if ((u64)base + (u64)cnt > (u64)max_entries) {
            atomicOr(&hdr->status, 1u << PL_CAPACITY_EXCEEDED);
            base_s = -1;
            tile_info[tile] = make_int2(0, 0);
        } else {
            base_s = (int)base;
            tile_info[tile] = make_int2((int)base, cnt);
        }
    }
    // the per-splat records do not need the tile's first global entry: they are written while thread
    // 0's atomic is in flight
    u16 lfin[PD + 1];
    u16* rec_tile = rec + (size_t)tile * SPLATS;
#pragma unroll
    for (int r = 0; r <= PD; r++) {
        lfin[r] = valid ? (u16)(seg[r] + lidx_s[get_rep(r)]) : (u16)0;   // the representative has the same remainder
        store_once(rec_tile + r * TP + tid, lfin[r]);
    }
    // The tile's splats sorted by entry (what the splat stage walks): a counting sort whose first half,
    // one shared-memory atomic per splat, returns the splat's place inside its entry's run.
    int place[PD + 1];
    if constexpr (SORTED) {
#pragma unroll
        for (int r = 0; r <= PD; r++) place[r] = valid ? atomicAdd(&run_s[lfin[r]], 1) : 0;
    }
    __syncthreads();
    // The next kernel may start when the tiles have ended, not before: with CTAs of clear_table coming while tiles still wrote their keys,
    // the insert behind it took half as long again on noisy images and points (5 x 300x300 28 -> 41 us, 10 of them 54 -> 80, 1.2 M different
    // keys in double 78 -> 96), however little either kernel had to do with it.  us a call: 400x400 of noise 241 -> 212, 2 x 512x512 x 6 of noisy images 982 ->
    // 891, 174x593 147 -> 133; photo, volumes and dense CRF 0.0 to 0.2 % more.
    const int base = base_s;
    if constexpr (COMPACT) {
        if (valid && base >= 0) {
#pragma unroll 1
            for (int r = 0; r <= PD; r++) {
                const int me = r * TP + tid;
                if (rep_s[me] == me) list_keys[(size_t)base + (seg[r] + lidx_s[me])] = TileKeys<PD>::template global_key<KW>(k.w, item);
                if (r < PD) k.step(r + 1);
            }
        }
    } else if (base >= 0) {
        // A thread an entry: its key, from the splat that owner_s names, and its bit in the sketch.  A tile has fewer
        // entries than threads, mostly; done by every splat that represents one, the same cost every warp a branch
        // a remainder, and the sketch a hash a splat.  With this and the cheaper floor and wrap of find_simplex, us a
        // call, forward + backward: two volumes of 111x128x120 549 -> 517, 1024x1024 grey by RGB 325 -> 309, 16 x 512x512
        // x 21 1823 -> 1794; 800x1200 x 3, forward, 188 -> 180.
        for (int e = tid; e < cnt; e += TP) {
            int r = 0, first = 0;
#pragma unroll
            for (int q = 1; q <= PD; q++) {
                r = e >= seg[q] ? q : r;
                first = e >= seg[q] ? seg[q] : first;
            }
            const int id = r * TP + owner_s[r * TP + e - first];
            u32 kw[Cfg<PD>::CW];
            keys.load(id, r, kw);
            list_keys[(size_t)base + e] = TileKeys<PD>::template global_key<KW>(kw, item);
            add_to_sketch(hdr, TileKeys<PD>::hash(kw, (u32)item * TILE_SEED), sketch_shift);
        }
    }
    if constexpr (SORTED && !is_double<R>::value) {
        // run starts: exclusive prefix sum of the entries' splat counts (thread t owns entries
        // t (PD+1) .. t (PD+1) + PD)
        const int lane = tid & 31, warp = tid >> 5;
        int local[PD + 1];
        int sum = 0;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int i = tid * (PD + 1) + r;
            local[r] = sum;
            sum += (i < cnt) ? run_s[i] : 0;
        }
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += t;
        }
        if (lane == 31) wsum_s[warp] = incl;
        __syncthreads();
        int before = 0;
#pragma unroll
        for (int q = 0; q < TP / 32; q++) before += (q < warp) ? wsum_s[q] : 0;
        const int excl = incl - sum + before;
#pragma unroll
        for (int r = 0; r <= PD; r++) {
            const int i = tid * (PD + 1) + r;
            if (i < cnt) run_s[i] = excl + local[r];
        }
        __syncthreads();
        // the list is assembled in shared memory (the key list is dead: the barriers above are behind every
        // thread's key stores) and leaves as one bulk copy
        uint2* sorted_s = reinterpret_cast<uint2*>(smem_raw);
        if (valid) {
            const R* recw_mine = rec_w + (size_t)tile * SPLATS + tid;   // this thread's own earlier stores
#pragma unroll
            for (int r = 0; r <= PD; r++) {
                const int pos = run_s[lfin[r]] + place[r];
                sorted_s[Cfg<PD>::srec_slot(pos)] =
                    make_uint2((unsigned)tid | ((unsigned)lfin[r] << 16), __float_as_uint(recw_mine[r * TP]));
            }
        }
        fence_async_proxy();
        __syncthreads();
        if (tid == 0) {
            bulk_store(srec + (size_t)tile * Cfg<PD>::SREC, sorted_s, (unsigned)(sizeof(uint2) * Cfg<PD>::SREC));
            bulk_store_finish();
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Table capacity, chosen on the device, a power of two: at least twice the entries (at least 1024), in calls that keep a sketch of
// the lattice's size at least four times the vertices it tells of if that is less (twice as many cost the probe chains of insert_entries
// more than the smaller table gained it), in a table of keys beyond 32 MB at least twice.
// clear_table: calls with a sketch (clear_header has cleared the table of all others).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ u32 log2_of_slots(u64 need, u32 max_log2) {
    u32 lg = 10;
    while (lg < max_log2 && (1ull << lg) < need) lg++;
    return lg;
}
constexpr u64 KEY_SLOTS_WHOLE = 1ull << 21;   // 32 MB
constexpr u64 TAG_SLOTS_WHOLE = 1ull << 23;   // 64 MB
constexpr u64 TAG_SLOTS_MOST = 1ull << 25;    // beyond, half as many would not stay in L2 either
constexpr float MOSTLY_NEW = 0.3f;            // vertices an entry, see insert_keys
template <bool KEY_SLOTS>
__global__ void __launch_bounds__(256)
clear_table(Header* hdr, u64* __restrict__ table, u32 max_log2, int sketch_shift) {
    after_previous_kernel();
    if (hdr->status != 0) return;
    __shared__ u32 bits_s[8];
    u64 need = 2ull * hdr->num_entries;
    bool mostly_new = false;
    if (need > (1ull << (sketch_shift + 10))) {
        const uint4* sketch = reinterpret_cast<const uint4*>(hdr + 1);
        u32 bits = 0;
#pragma unroll
        for (int i = 0; i < SKETCH_WORDS / 4 / 256; i++) {
            const uint4 v = sketch[i * 256 + threadIdx.x];
            bits += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
        bits = __reduce_add_sync(0xFFFFFFFFu, bits);
        if ((threadIdx.x & 31) == 0) bits_s[threadIdx.x >> 5] = bits;
        __syncthreads();
        u32 set = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) set += bits_s[i];
        // Distinct sampled keys: -B ln(share of bits still clear).  With 2^10 or more of them the error of the
        // estimate stays below 4 % (one standard deviation), far from the factor by which the table is larger;
        // with fewer there are at most about 2^(shift + 10) vertices, for which the smallest table has room.
        const u32 clear = (1u << SKETCH_LOG2) - set;
        if (clear > (1u << SKETCH_LOG2) / 64) {
            const float sampled = -(float)(1 << SKETCH_LOG2) * logf((float)clear * (1.f / (1 << SKETCH_LOG2)));
            const float vertices = sampled * (float)(1u << sketch_shift);
            mostly_new = vertices >= MOSTLY_NEW * (float)hdr->num_entries;
            u64 slots = (u64)(4.f * vertices);
            // four a vertex spare more probes than the larger table costs while it stays in L2 beside everything else; a
            // table of keys beyond 32 MB has two a vertex at least (us a call, four / two a vertex: 1024x1024 grey by RGB,
            // forward + backward, 17 MB at four, 325 / 337; 16 x 512x512 x 21, 67 MB at four, 1857 / 1824.  So has
            // a tagged one beyond 64 MB (1 M points, pd 16, 134 / 67 MB with keys of one sector: insert 454 / 404 us, link
            // 670 / 578, clear 31 / 18; 4 x 300x300 points 1775 / 1447 us a call), up to 256 MB (8 M points, 16 M vertices, 13.5 / 13.8 ms
            // of index)
            constexpr u64 WHOLE = KEY_SLOTS ? KEY_SLOTS_WHOLE : TAG_SLOTS_WHOLE;
            if (slots > WHOLE && (KEY_SLOTS || slots <= TAG_SLOTS_MOST)) slots = slots / 2 > WHOLE ? slots / 2 : WHOLE;
            const u64 least = 1ull << (sketch_shift + 11);
            slots = slots < least ? least : slots;
            need = slots < need ? slots : need;
        }
    }
    const u32 lg = log2_of_slots(need, max_log2);
    const u32 filter_log2 =
        (!KEY_SLOTS && lg >= FILTER_MIN_LOG2 && lg < max_log2) ? min(lg + FILTER_BITS_LOG2, FILTER_MAX_LOG2) : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        hdr->table_log2 = lg;
        hdr->filter_log2 = filter_log2;
        hdr->mostly_new = mostly_new && (1ull << lg) <= KEY_SLOTS_WHOLE ? 1u : 0u;
    }
    if constexpr (!KEY_SLOTS) {
        if (filter_log2) {
            uint4* filter = reinterpret_cast<uint4*>(filter_words(table, max_log2, filter_log2));
            for (u64 i = grid_thread(); i < (1ull << (filter_log2 - 7)); i += grid_threads())
                filter[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    const u64 cap = 1ull << lg;
    for (u64 i = grid_thread(); i < cap; i += grid_threads()) {
        if constexpr (KEY_SLOTS) reinterpret_cast<ulonglong2*>(table)[i] = make_ulonglong2(EMPTY_SLOT, EMPTY_SLOT);
        else table[i] = EMPTY_SLOT;
    }
}

// ---------------------------------------------------------------------------------------------
// insert_entries
// ---------------------------------------------------------------------------------------------
// The items that the lattice serves (1, or see one_for_all), and their value rows, to be zeroed: a vertex's together, item by item, so that
// to the blur, the conversion of the fixed-point sums and the zeroing they are one long row, or an item's together, in large lattices (see
// rows_together).
struct ItemRows {
    u32 items, stride;         // entries from one item's to the next's
    u32 row_step, item_step;   // rows from a vertex's to the next's, and from an item's to the next's
    uint4* rows;               // float rows, rows of doubles, or the 64-bit sums of the deterministic mode; null: none
    u32 row_quads;             // 16 bytes each
};
__device__ __forceinline__ void zero_rows_of(const ItemRows& z, u32 M, u32 thread, u32 threads) {
    if (!z.rows) return;
    const u64 quads = (u64)M * z.row_step * z.row_quads;
    if (z.item_step <= 1) {
        for (u64 i = thread; i < quads; i += threads) z.rows[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    // quads of every item, one stretch after another
    if (quads == 0) return;
    const u32 fit = quads <= threads ? (u32)quads : 0u;   // (else a step stays within two items)
    const u32 items_on = fit ? threads / fit : 0u, on = threads - items_on * fit;
    u32 b = fit ? thread / fit : 0u;
    u64 i = thread - b * fit;
    while (b < z.items) {
        z.rows[(u64)b * z.item_step * z.row_quads + i] = make_uint4(0u, 0u, 0u, 0u);
        b += items_on;
        i += on;
        if (i >= quads) {
            i -= quads;
            b++;
        }
    }
}
// Calls store(t, b, vertex) for the T entries of every item b, where find(t) is an entry's vertex.  A thread goes through the items of its
// entry, which it looks up once, while an eighth of the threads have one; fewer entries are spread over all threads (16x300x300, 200 k
// entries of 303 k threads, 137 / 142 us a call).  (Their number in all items fits 31 bits, as the bound does.)
template <typename Find, typename Store>
__device__ __forceinline__ void for_entries_of(const ItemRows& z, u32 T, u32 thread, u32 threads, Find find, Store store) {
    if (z.items == 1 || T >= threads / 8) {
        for (u32 t = thread; t < T; t += threads) {
            const u32 v = find(t);
            for (u32 b = 0; b < z.items; b++) store(t, b, v);
        }
        return;
    }
    const u32 all = T * z.items;
    for (u32 i = thread; i < all; i += threads) {
        const u32 b = i / T, t = i - b * T;
        store(t, b, find(t));
    }
}
// Entry t of item b has vertex v: the row that is its, in that item's copy of the list.
__device__ __forceinline__ void store_vertex_of(const ItemRows& z, u32* list_ref, u32 t, u32 b, u32 v) {
    list_ref[b * z.stride + t] = v * z.row_step + b * z.item_step;
}

// What the insert launch sets up for every vertex it creates, so that no later launch has to: the
// vertex's key (vertex order) and its slots of the neighbour table ("missing").  (Its value row is zeroed by the link launch,
// by streaming stores under the latency of its lookups.)
struct VertexInit {
    int* nbr;            // [pd + 1][max_entries] pairs
    u64 max_entries;
    int pd;
};

// Entries are inserted in rounds of INSERT_CHUNKS chunks of 256: the winners of a round (entries that
// created a vertex) are collected in shared memory and numbered with ONE atomic on the global vertex
// counter.  One atomic per chunk, all on the same address, was what bounded this launch.
constexpr int INSERT_CHUNKS = 8;

// The table's size in calls whose clear_header cleared all that the table may take: by the entries, here; else clear_table
// has chosen it (see there).  By all threads of an insert launch alike; one of them tells the lookups after it.
__device__ __forceinline__ u32 table_log2_of(Header* hdr, u32 entries, u32 max_log2, bool cleared) {
    if (!cleared) return hdr->table_log2;
    const u32 lg = log2_of_slots(2ull * entries, max_log2);
    if (blockIdx.x == 0 && threadIdx.x == 0) hdr->table_log2 = lg;
    return lg;
}
constexpr u32 VERTEX_FLAG = 0x80000000u;   // low word of a table slot: vertex index (set) or entry index (clear)

struct InsertRound {
    u32 t[INSERT_CHUNKS * 256];      // winners of the round: entry ...
    u32 slot[INSERT_CHUNKS * 256];   // ... and the table slot it claimed
    u32 count, base;
};

// Appends a winner to the round's list; one shared-memory atomic per warp.
__device__ __forceinline__ void round_add_winner(InsertRound& rd, bool winner, u32 t, u32 slot) {
    const unsigned ballot = __ballot_sync(0xFFFFFFFFu, winner);
    if (!ballot) return;
    const int lane = threadIdx.x & 31, leader = __ffs(ballot) - 1;
    u32 first = 0;
    if (lane == leader) first = atomicAdd(&rd.count, (u32)__popc(ballot));
    first = __shfl_sync(0xFFFFFFFFu, first, leader);
    if (winner) {
        const u32 pos = first + __popc(ballot & ((1u << lane) - 1u));
        rd.t[pos] = t;
        rd.slot[pos] = slot;
    }
}

// Ends a round: numbers its winners (consecutive vertex indices), writes vid and the vertex-ordered keys,
// initialises the new vertices, and re-labels the winners' table slots with the vertex index, so that a
// lookup ends at the slot (tag, vertex) and the vertex's key instead of walking entry -> owner -> vertex.
// `relabel` writes the slot, whole, that a key claimed for vertex v: BEHIND_KEYS with the upper half of the key's hash, when
// the keys of the round are visible, which lookups of this launch compare (tagged slots); else with the key.  Called by all threads.
template <bool BEHIND_KEYS, int KW, typename Relabel>
__device__ __forceinline__ void finish_round(Header* hdr, InsertRound& rd, const Key<KW>* __restrict__ list_keys,
                                             u32* __restrict__ vid, Key<KW>* __restrict__ vkeys,
                                             const VertexInit& vi, Relabel relabel) {
    __syncthreads();
    if (threadIdx.x == 0) rd.base = rd.count ? atomicAdd(&hdr->num_vertices, rd.count) : 0u;
    __syncthreads();
    const u32 base = rd.base, tot = rd.count;
    for (u32 i = threadIdx.x; i < tot; i += 256) {
        const u32 t = rd.t[i], v = base + i;
        const Key<KW> k = list_keys[t];
        vid[t] = v;
        vkeys[v] = k;
        if constexpr (BEHIND_KEYS) rd.t[i] = (u32)(hash_key<KW>(k) >> 32);   // (read again by this thread alone)
        else relabel(rd.slot[i], k, v);
    }
    if constexpr (BEHIND_KEYS) {
        if (tot) __threadfence();   // a key is visible before its slot says "vertex v"
        for (u32 i = threadIdx.x; i < tot; i += 256) relabel(rd.slot[i], rd.t[i], base + i);
    }
    if (tot) {
        int2* nb = reinterpret_cast<int2*>(vi.nbr);
        for (int a = 0; a <= vi.pd; a++)
            for (u32 i = threadIdx.x; i < tot; i += 256) store_once(nb + (u64)a * vi.max_entries + base + i, make_int2(-1, -1));
    }
    __syncthreads();
    if (threadIdx.x == 0) rd.count = 0;
    __syncthreads();
}

// A table slot holds (32-bit hash tag, index): the index of the vertex once its creator's round has ended
// (VERTEX_FLAG set; full key in vkeys), before that the index of the entry that created it (full key in
// list_keys, which the previous launch has completely written).
template <int KW>
__global__ void __launch_bounds__(256)
insert_entries(Header* hdr, u64* __restrict__ table, u32 max_log2, const Key<KW>* __restrict__ list_keys,
               u32* __restrict__ list_ref, u32* __restrict__ vid, Key<KW>* __restrict__ vkeys, VertexInit vi, bool cleared) {
    wait_for_previous_kernel();
    __shared__ InsertRound rd;
    if (threadIdx.x == 0) rd.count = 0;
    if (call_failed(hdr)) return;   // (its barrier also publishes rd.count)
    const u32 T = hdr->num_entries;
    const u64 mask = (1ull << table_log2_of(hdr, T, max_log2, cleared)) - 1;
    const u32 filter_log2 = hdr->filter_log2;
    u32* filter = filter_log2 ? filter_words(table, max_log2, filter_log2) : nullptr;
    const u32 stride = gridDim.x * 256u;
    for (u32 start = blockIdx.x * 256u; start < T;) {
        for (int c = 0; c < INSERT_CHUNKS && start < T; c++, start += stride) {
            const u32 t = start + threadIdx.x;
            bool winner = false;
            u64 my_slot = 0;
            if (t < T) {
                const Key<KW> k = load_key_once<KW>(list_keys + t);
                const u64 h = hash_key<KW>(k);
                const u64 mine = (h & 0xFFFFFFFF00000000ull) | (u64)t;
                u32 ref = 0xFFFFFFFFu;
                // probe; on an empty slot try to claim it, and keep probing from there if another entry was faster
                u64 s = h & mask;
                for (u64 it = 0; it <= mask; it++) {
                    // slots and vertex keys change during this launch: read them from L2, never from an
                    // L1 line that may predate another CTA's write
                    u64 cur = load_relaxed(&table[s]);
                    if (cur == EMPTY_SLOT) {
                        cur = atomicCAS(&table[s], EMPTY_SLOT, mine);
                        if (cur == EMPTY_SLOT) {
                            ref = t;
                            winner = true;
                            my_slot = s;
                            if (filter) {
                                const u32 bit = (u32)h & ((1u << filter_log2) - 1u);
                                atomicOr(filter + (bit >> 5), 1u << (bit & 31u));
                            }
                            break;
                        }
                    }
                    if ((u32)(cur >> 32) == (u32)(h >> 32)) {
                        const u32 low = (u32)cur;
                        const Key<KW> other = (low & VERTEX_FLAG) ? load_key_l2<KW>(&vkeys[low & ~VERTEX_FLAG])
                                                                  : list_keys[low];
                        if (key_equal<KW>(other, k)) { ref = low; break; }
                    }
                    s = (s + 1) & mask;
                }
                if (ref == 0xFFFFFFFFu) {
                    atomicOr(&hdr->status, 1u << PL_INTERNAL_ERROR);
                    ref = t;
                }
                store_once(list_ref + t, ref);   // owning entry, or (VERTEX_FLAG set) the vertex itself
            }
            round_add_winner(rd, winner, t, (u32)my_slot);
        }
        finish_round<true, KW>(hdr, rd, list_keys, vid, vkeys, vi, [&](u32 slot, u32 tag, u32 v) {
            store_relaxed(table + slot, ((u64)tag << 32) | VERTEX_FLAG | v);
        });
    }
}

// Table of keys (pd up to 5): a slot of 16 bytes holds the key itself, four fields in its first word, the others above
// the index in its second, so that a lookup is one access to a random sector and not one to the slot and one to the key
// it names: the index kernels run at the rate of such accesses.  link_neighbours on 800x1200 x 3: 34.5 -> 30.1 us, on
// 16 x 512x512: 69 -> 63 (a neighbour that is there costs one access and not two); insert_entries a few per cent, where
// entries come in duplicates whose key was in L2 already.
struct alignas(16) KeySlot { u64 first, rest; };   // rest: other fields << 32 | index (as in a slot of 8 bytes); all ones: empty
__device__ __forceinline__ KeySlot load_slot(const KeySlot* p) {   // from L2, in one piece
    KeySlot s;
    asm volatile("{\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%2];\n\tmov.b128 {%0, %1}, v;\n\t}"
                 : "=l"(s.first), "=l"(s.rest)
                 : "l"(p)
                 : "memory");
    return s;
}
__device__ __forceinline__ void store_slot(KeySlot* p, u64 first, u64 rest) {
    asm volatile("{\n\t.reg .b128 v;\n\tmov.b128 v, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p), "l"(first), "l"(rest)
                 : "memory");
}
// Writes the key to an empty slot; what was there.
__device__ __forceinline__ KeySlot claim_slot(KeySlot* p, u64 first, u64 rest) {
    KeySlot s;
    asm volatile("{\n\t.reg .b128 empty, mine, was;\n\tmov.b128 empty, {%3, %3};\n\tmov.b128 mine, {%4, %5};\n\t"
                 "atom.relaxed.gpu.global.cas.b128 was, [%2], empty, mine;\n\tmov.b128 {%0, %1}, was;\n\t}"
                 : "=l"(s.first), "=l"(s.rest)
                 : "l"(p), "l"(EMPTY_SLOT), "l"(first), "l"(rest)
                 : "memory");
    return s;
}
template <int PD>
__device__ __forceinline__ u32 key_rest(const Key<Cfg<PD>::KW>& k) {
    constexpr int KW = Cfg<PD>::KW;
    return KW > 1 ? (u32)k.w[KW - 1] : 0u;
}

// insert_entries into a table of keys.  The index in a slot is that of the creating entry, then (its round ended) of
// the vertex.
// A compare-and-swap on a line that was just read takes longer than one on a line that was not: in a table of 32 MB a ns sees 175 loads of
// random slots, 80 swaps, 50 times load, swap and store of an empty slot, 70 times swap and store.  So slots are claimed unseen where the sketch
// says that MOSTLY_NEW of the entries or more are vertices and the table stays in L2 (up to 32 MB; beyond, the load brings the line in for the
// swap).  us a call, a look first / not, by the share of vertices, below the line 14 %, 8 x 512x512 x 3 251 / 255, 19 % 225 / 226, 24 %, 4 x
// 512x512 x 3
// 148 / 147, 30 %, 1024x1024 x 3 121 / 120, but 2 x 111x128x120 of a noisy guide, 20 to 30 %, 423 / 432; above it 1024x1024 x 3, 31 % 122 / 122,
// 34 % 162
// / 159, 39 % 238 / 236, 800x1200 x 3, 52 % 155 / 152, 57 % 206 / 203.  Tables of 64 MB and more: 8 x 512x512 x 3, noise 0.16, 730 / 755, 0.25
// 1166 / 1193, 800x1200 x 3, 73 %, 714 / 720.
// In calls without a sketch a warp does as long as a third of what it claims is free, which the first of the entries mostly are, whatever
// the lattice: 300x400 x 3, 29 % 36 / 36, 32 % 41.4 / 40.3, 35 % 44 / 42.6, 40 % 56 / 54.5, 46 % 80.7 / 80.9, 512x512 x 3, 51 % 55.7 / 54.7, 63 %
// 99.6 / 100.
template <int PD>
__global__ void __launch_bounds__(256, 8)   // as many as it is launched with
insert_keys(Header* hdr, KeySlot* __restrict__ table, u32 max_log2, const Key<Cfg<PD>::KW>* __restrict__ list_keys,
            u32* __restrict__ list_ref, u32* __restrict__ vid, Key<Cfg<PD>::KW>* __restrict__ vkeys, VertexInit vi, bool cleared) {
    wait_for_previous_kernel();
    constexpr int KW = Cfg<PD>::KW;
    __shared__ InsertRound rd;
    if (threadIdx.x == 0) rd.count = 0;
    if (call_failed(hdr)) return;   // (its barrier also publishes rd.count)
    const u32 T = hdr->num_entries;
    const u32 mask = (u32)((1ull << table_log2_of(hdr, T, max_log2, cleared)) - 1);
    const u32 stride = gridDim.x * 256u;
    bool unseen = cleared || hdr->mostly_new != 0;
    // entry t, of which slot s of the table is the first to ask; true: it has claimed slot s
    auto insert = [&](auto unseen_too, u32 t, u32& s) -> bool {
        const Key<KW> k = list_keys[t];
        const u64 first = k.w[0];
        const u32 rest = key_rest<PD>(k);
        u32 ref = 0xFFFFFFFFu;
        bool winner = false;
        s = (u32)hash_key<KW>(k) & mask;
        for (u64 it = 0; it <= mask; it++) {
            KeySlot cur = {EMPTY_SLOT, EMPTY_SLOT};
            if constexpr (!decltype(unseen_too)::value) cur = load_slot(table + s);
            if ((u32)cur.rest == 0xFFFFFFFFu) {
                cur = claim_slot(table + s, first, ((u64)rest << 32) | t);
                if ((u32)cur.rest == 0xFFFFFFFFu) {
                    ref = t;
                    winner = true;
                    break;
                }
            }
            if (cur.first == first && (u32)(cur.rest >> 32) == rest) { ref = (u32)cur.rest; break; }
            s = (s + 1) & mask;
        }
        if (ref == 0xFFFFFFFFu) {
            atomicOr(&hdr->status, 1u << PL_INTERNAL_ERROR);
            ref = t;
        }
        list_ref[t] = ref;   // owning entry, or (VERTEX_FLAG set) the vertex itself
        return winner;
    };
    for (u32 start = blockIdx.x * 256u; start < T;) {
        for (int c = 0; c < INSERT_CHUNKS && start < T; c++, start += stride) {
            const u32 t = start + threadIdx.x;
            bool winner = false;
            u32 s = 0;
            if (unseen) {
                if (t < T) winner = insert(std::true_type{}, t, s);
            } else {
                if (t < T) winner = insert(std::false_type{}, t, s);
            }
            round_add_winner(rd, winner, t, s);
            if (cleared) unseen = 3 * __popc(__ballot_sync(0xFFFFFFFFu, winner)) >= 32;
        }
        finish_round<false, KW>(hdr, rd, list_keys, vid, vkeys, vi, [&](u32 slot, const Key<KW>& k, u32 v) {
            store_slot(table + slot, k.w[0], ((u64)key_rest<PD>(k) << 32) | VERTEX_FLAG | v);
        });
    }
}

// entry -> vertex: after the insert launch owners[t] names the entry that owns t's key; the link launch turns that into the
// owner's vertex index, in list_ref (first loop of link_neighbours / link_neighbours_direct).  The two are the same memory
// where the lattice serves one item.
__device__ __forceinline__ void resolve_entries(const Header* hdr, const u32* owners, u32* list_ref,
                                                const u32* __restrict__ vid, const ItemRows& rows) {
    for_entries_of(
        rows, hdr->num_entries, (u32)grid_thread(), (u32)grid_threads(),
        [&](u32 t) {
            const u32 ref = owners[t];
            return (ref & VERTEX_FLAG) ? (ref & ~VERTEX_FLAG) : vid[ref];
        },
        [&](u32 t, u32 b, u32 v) { store_vertex_of(rows, list_ref, t, b, v); });
}

// ---------------------------------------------------------------------------------------------
// link_neighbours: entry -> vertex, then the +-1 neighbours of every vertex along each of the PD+1
// lattice axes.
// ---------------------------------------------------------------------------------------------
// One table lookup per (vertex v, axis a): the neighbour u whose key is v's key with every stored
// coordinate +1, except coordinate a which moves by -PD (along axis PD no stored coordinate is
// special; src/PermutohedralLatticeCPU.h:381-388).  Then u is v's "+" neighbour and v is u's "-"
// neighbour, so the second lookup of the reference is not needed.
// One thread per (vertex, axis), axis = blockIdx.y: neighbouring threads take neighbouring vertices of one axis,
// so their key loads and their own slots of the neighbour table are contiguous.  The neighbour's key and the
// linear part of its hash differ from the vertex's by constants of the axis.  Every slot carries a vertex index by
// now, so a lookup is two dependent accesses, and one where there is no neighbour.  (One thread for all axes of a
// vertex, its first probes in flight together, took up to twice as long: its key comparisons wait for one another.)
template <int PD>
__host__ __device__ constexpr u64 axis_word(int a, int j) {   // what moving along axis a adds to key word j
    return coord_ones<PD>(j) - ((a < PD && (a >> 2) == j) ? (u64)(PD + 1) << (16 * (a & 3)) : 0ull);
}
template <int PD>
__host__ __device__ constexpr u64 axis_hash(int a) {          // and to its linear hash
    u64 h = 0;
    for (int j = 0; j < Cfg<PD>::KW; j++) h += axis_word<PD>(a, j) * hash_factor(j);
    return h;
}
template <int PD, int KW, int A>
__device__ __forceinline__ void link_axis(const u64* __restrict__ table, u64 mask, const u32* __restrict__ filter,
                                          u32 filter_mask,
                                          const Key<KW>* __restrict__ vkeys, u32 M, int* __restrict__ nbr,
                                          u64 max_entries) {
    int* __restrict__ nbr_axis = nbr + 2 * (u64)A * max_entries;
    for (u32 v = blockIdx.x * blockDim.x + threadIdx.x; v < M; v += gridDim.x * blockDim.x) {
        Key<KW> k = vkeys[v];
        const u64 h = mix_hash(linear_hash<KW>(k) + axis_hash<PD>(A));
        if (filter) {
            const u32 bit = (u32)h & filter_mask;
            if (!((__ldg(filter + (bit >> 5)) >> (bit & 31u)) & 1u)) continue;
        }
#pragma unroll
        for (int j = 0; j < KW; j++) k.w[j] += axis_word<PD>(A, j);
        u64 s = h & mask;
        for (u64 it = 0; it <= mask; it++) {
            const u64 cur = table[s];
            if (cur == EMPTY_SLOT) break;
            if ((u32)(cur >> 32) == (u32)(h >> 32)) {
                const u32 u = (u32)cur & ~VERTEX_FLAG;
                if (key_equal<KW>(vkeys[u], k)) {
                    store_once(nbr_axis + 2 * (u64)v, (int)u);
                    store_once(nbr_axis + 2 * (u64)u + 1, (int)v);
                    break;
                }
            }
            s = (s + 1) & mask;
        }
    }
}
// The same in a table of keys.
template <int PD, int KW, int A>
__device__ __forceinline__ void link_axis(const KeySlot* __restrict__ table, u32 mask,
                                          const Key<KW>* __restrict__ vkeys, u32 M, int* __restrict__ nbr,
                                          u64 max_entries) {
    int* __restrict__ nbr_axis = nbr + 2 * (u64)A * max_entries;
    for (u32 v = blockIdx.x * blockDim.x + threadIdx.x; v < M; v += gridDim.x * blockDim.x) {
        Key<KW> k = vkeys[v];
        u32 s = (u32)mix_hash(linear_hash<KW>(k) + axis_hash<PD>(A)) & mask;
#pragma unroll
        for (int j = 0; j < KW; j++) k.w[j] += axis_word<PD>(A, j);
        for (u64 it = 0; it <= mask; it++) {
            const ulonglong2 cur = __ldg(reinterpret_cast<const ulonglong2*>(table + s));
            if ((u32)cur.y == 0xFFFFFFFFu) break;
            if (cur.x == k.w[0] && (u32)(cur.y >> 32) == key_rest<PD>(k)) {
                const u32 u = (u32)cur.y & ~VERTEX_FLAG;
                store_once(nbr_axis + 2 * (u64)v, (int)u);
                store_once(nbr_axis + 2 * (u64)u + 1, (int)v);
                break;
            }
            s = (s + 1) & mask;
        }
    }
}
template <int PD, int KW, int A>
struct LinkAxis {   // link_axis of the axis this block works on, chosen once per block
    template <typename... Args>
    __device__ static __forceinline__ void run(int axis, Args... args) {
        if (axis == A)
            link_axis<PD, KW, A>(args...);
        else if constexpr (A < PD)
            LinkAxis<PD, KW, A + 1>::run(axis, args...);
    }
};

template <int PD, bool KEY_SLOTS, int KW = Cfg<PD>::KW>
__global__ void __launch_bounds__(256)
link_neighbours(Header* hdr, u64* __restrict__ table, u32 max_log2, const u32* owners, u32* list_ref,
                const u32* __restrict__ vid, const Key<KW>* __restrict__ vkeys, int* __restrict__ nbr,
                u64 max_entries, ItemRows rows, Watch watch) {
    after_previous_kernel();
    report_to(watch, hdr);
    if (hdr->status != 0) return;
    resolve_entries(hdr, owners, list_ref, vid, rows);
    const u32 M = hdr->num_vertices;
    const u64 mask = (1ull << hdr->table_log2) - 1;
    zero_rows_of(rows, M, (u32)grid_thread(), (u32)grid_threads());   // under the latency of the lookups below
    if constexpr (KEY_SLOTS) {
        LinkAxis<PD, KW, 0>::run((int)blockIdx.y, reinterpret_cast<const KeySlot*>(table), (u32)mask, vkeys, M, nbr, max_entries);
    } else {
        const u32 filter_log2 = hdr->filter_log2;
        const u32* filter = filter_log2 ? filter_words(table, max_log2, filter_log2) : nullptr;
        LinkAxis<PD, KW, 0>::run((int)blockIdx.y, table, mask, filter, (1u << filter_log2) - 1u, vkeys, M, nbr, max_entries);
    }
}

}  // namespace pl
