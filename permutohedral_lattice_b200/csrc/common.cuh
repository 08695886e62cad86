// Shared definitions of the lattice kernels: geometry of a call, workspace header and layout, packed
// vertex keys and their hashes, tile addressing, vector reductions and asynchronous-copy helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/pl_lattice.h"
#include "simplex.cuh"

namespace pl {

typedef unsigned long long u64;
typedef unsigned int u32;
typedef unsigned short u16;

constexpr u64 EMPTY_SLOT = ~0ull;
constexpr int MAX_SDIMS = 8;
constexpr int MAX_PD = 16;

// ---------------------------------------------------------------------------------------------
// Geometry of a call: how points map to tiles and how features are produced.
// ---------------------------------------------------------------------------------------------
struct Geom {
    int batch, n;           // items, points per item
    int W, H, outer;        // n = outer * H * W (W fastest)
    int TX, TY;             // tile = TY rows of TX points, TX * TY = TP
    int tiles_x, tiles_y, tiles_per_item, num_tiles;
    int tx_log2;            // TX is a power of two
    int grid3;              // 1: tile kernels run on a (tiles_x, tiles_y, batch * outer) grid
    int n_sdims, R;         // op path: spatial dims and reference channels (pd = n_sdims + R)
    int sdims[MAX_SDIMS];
    float spatial_std, feature_std;
    float spatial_rcp, feature_rcp;   // correctly rounded reciprocals of the two (host-computed)
    int rcp_div;            // 1: divide through the reciprocals (exact for these operands), 0: IEEE divide
    int calm_entries;       // entries of a tile up to which its points hardly change entry in disorder (see ColumnsSample)
    int from_positions;     // 1: features are read from a positions array
    int lattice_items;      // items that one lattice serves (see one_for_all): records and vertices are those of item 0
    u32 item_entries;       // then: entries from one item's to the next's
    u32 row_step;           // value rows from a vertex's to the next's: the items where theirs lie together (see ItemRows), else 1
    u32 bound;              // then: the call's max_entries (the lattice's own is a share of it)
    float scale[MAX_PD];    // host-computed scale factors (double arithmetic rounded to float)
    // T = double calls: the same three in double
    double spatial_std_d, feature_std_d;
    double scale_d[MAX_PD];
};

struct Header {   // first 256 bytes of the workspace
    u32 num_entries;
    u32 num_vertices;
    u32 status;
    u32 table_log2;
    u32 absmax_bits;   // deterministic mode: bit pattern of max |input| (non-negative floats order as integers)
    u32 direct;        // 1: vertices were found by direct indexing (spatial-only call), 0: through the hash table
    u32 capacity;      // the max_entries the workspace was laid out for (written by build_tiles)
    u32 sorted;        // 1: the lattice was built for reuse and holds every tile's splats sorted by entry
    u32 filter_log2;   // bits of the vertex filter behind the table, as a logarithm; 0: none (see FILTER_BITS_LOG2)
    u32 reported;      // status bits that the call's watch has told the host of (see Watch)
    u32 calm_entries;  // of the Geom that the lattice was built with
    u32 items;         // items that the lattice serves: entries and vertices are those of one of them
    u32 mostly_new;    // in calls with a sketch: 30 % of the entries or more are vertices, in a table that stays in L2 (see insert_keys)
    u32 row_step;      // of the Geom that the lattice was built with
    u32 pad[50];
};

// Sketch of the lattice's size, behind the header (zeroed with it): a bitmap in which build_tiles sets one bit
// for every key whose hash falls into a 2^-shift part of the hash range.  The bits set tell clear_table how many
// DISTINCT keys there are (linear counting), so that the table is sized by vertices and not by entries, of which
// there are up to 40 times as many.  The shift keeps the bitmap at most about half full in the worst case.
constexpr int SKETCH_LOG2 = 16;
constexpr int SKETCH_WORDS = (1 << SKETCH_LOG2) / 32;

// Filter in front of a large hash table: 2^FILTER_BITS_LOG2 bits a slot, one set for every vertex (by its key's hash).
// Most neighbour lookups of a sparse lattice find nothing; a table that does not stay in L2 costs each of them an
// access to DRAM, the filter, an eighth of its size, one to L2, and it lets few pass (a table has two to eight slots
// a vertex).  It lies at the end of the table's region, which has room for it whenever the table uses at most half of
// that, and is kept for tables of 2^FILTER_MIN_LOG2 slots (64 MB) and more; beyond 2^FILTER_MAX_LOG2 bits (32 MB) it
// would not stay in L2 itself.  1 M points with 16 features: 2133 ->
// 2044 us a call; with a table of 32 MB, which stays in L2, it cost one per cent (16 x 512x512 x 21, while pd 5 still had
// slots of 8 bytes).  Tables whose slots hold the key have none: a lookup there is one access anyway.
constexpr u32 FILTER_BITS_LOG2 = 3, FILTER_MIN_LOG2 = 23, FILTER_MAX_LOG2 = 28;
__device__ __forceinline__ u32* filter_words(u64* table, u32 max_log2, u32 filter_log2) {
    return reinterpret_cast<u32*>(table + (1ull << max_log2)) - (1ull << (filter_log2 - 5));
}

// Number of this thread in a grid of one or two dimensions, and how many there are.
__device__ __forceinline__ u64 grid_thread() {
    return (u64)(blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ u64 grid_threads() { return (u64)gridDim.x * gridDim.y * blockDim.x; }

// Where a watched call reports (pl_watch_next_call): two words of mapped host memory.  The link kernel writes
// sequence << 40 | status bits << 32 | entries into the first before it does anything else: whether the lattice fits,
// and whether it could be built, is known by then, and the host, which polls the word, goes on while the device still
// splats, blurs and slices.  What fails after that (the splat's bounded wait for its copies) the slice kernel, which
// then fills the output with NaN, writes into the second word; the host looks there when it watches again.
constexpr u32 WATCH_SEQ_MASK = 0xFFFFFFu;
struct Watch {
    u64* words;   // null: nobody is watching
    u32 seq;
};
__device__ __forceinline__ void store_to_host(u64* word, u64 v) {
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(word), "l"(v) : "memory");
}
__device__ __forceinline__ void report_to(const Watch& w, Header* hdr) {
    if (w.words && grid_thread() == 0) {
        const u32 status = __ldcg(&hdr->status);
        hdr->reported = status;
        store_to_host(w.words, ((u64)w.seq << 40) | ((u64)(status & 0xFFu) << 32) | (u64)(hdr->num_entries * hdr->items));
    }
}
// By the first thread of the grid of a slice kernel that has found the call failed.
__device__ __forceinline__ void report_late(const Watch& w, const Header* hdr) {
    if (w.words && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
        const u32 late = hdr->status & ~hdr->reported;
        if (late) store_to_host(w.words + 1, late);
    }
}

struct Layout {   // byte offsets into the workspace
    size_t tile_info, rec, rec_w, srec, list_keys, list_ref, vid, vkeys, table, nbr, v0, v1, v64, total;
    u64 max_entries;   // capacity of entry- and vertex-indexed arrays
    u64 table_slots;   // allocated slots (power of two)
    bool key_slots;    // they hold the key and take 16 bytes (see KeySlot); else 8
    u64 index_words;   // 32-bit words of the table's region that direct indexing may use
};

template <int KW>
struct alignas((KW % 2 == 0) ? 16 : 8) Key {
    u64 w[KW];
};

template <int PD>
struct Cfg {
    static constexpr int KW = (PD + 1 + 3) / 4;          // 16-bit fields: PD coordinates + item
    // Keys of a call of one item, where they need no item: 16 coordinates then fill one 32-byte sector, and comparing with
    // a key somewhere in the list touches one and not two (1 M points: insert 524 -> 454 us, build 279 -> 267).
    static constexpr int KW_ALONE = PD == 16 ? 4 : KW;
    static constexpr bool KEY_SLOTS = PD <= 5;           // a key and an index fit 16 bytes: see KeySlot
    static constexpr int TP = (PD <= 8) ? 256 : 128;     // points per tile = threads per CTA
    static constexpr int SPLATS = TP * (PD + 1);
    // 16-bit slots of the tile's hash: at least 2.5 per splat
    static constexpr int LSLOG = (5 * SPLATS <= 2 * 2048)    ? 11
                                 : (5 * SPLATS <= 2 * 4096)  ? 12
                                 : (5 * SPLATS <= 2 * 8192)  ? 13
                                                             : 14;
    static constexpr int LS = 1 << LSLOG;
    static_assert(5 * SPLATS <= 2 * LS && SPLATS <= 65535, "slots hold 16-bit splat numbers");
    // The tile's splats sorted by entry, as build_tiles leaves them for the splat kernels: cut into windows
    // of WL splats, each followed by two spare 8-byte words: lanes that walk neighbouring windows in step read two
    // splats at once, and windows an odd number of 16-byte words apart do not collide on shared-memory banks.  SREC
    // words per tile (even: the list moves by bulk copies, whose sizes are multiples of 16 bytes).
    static constexpr int WL = 8 * (PD + 1);
    static constexpr int SREC = SPLATS + 2 * (SPLATS / WL);
    __host__ __device__ static constexpr int srec_slot(int pos) { return pos + 2 * (pos / WL); }
    // What build_tiles keeps of the keys in shared memory (see TileKeys): every splat's key up to pd = 8, one
    // record per point above (a key of 16 coordinates for each of 17 splats would leave room for two CTAs an SM).
    static constexpr bool COMPACT = PD > 8;
    static constexpr int CW = (PD + 1) / 2;                                  // 32-bit words of two coordinates
    static constexpr int KEY_WORDS = COMPACT ? CW + 4 : CW <= 2 ? CW : 4;    // words of one key (point record)
    // build_tiles assembles the sorted list in the memory of its keys, which is therefore at least as large
    static constexpr size_t KEY_BYTES = sizeof(u32) * (size_t)KEY_WORDS * (COMPACT ? TP : SPLATS);
    __host__ __device__ static constexpr size_t build_keys(bool sorted) {
        return sorted && sizeof(uint2) * SREC > KEY_BYTES ? sizeof(uint2) * SREC : KEY_BYTES;
    }
    __host__ __device__ static constexpr size_t build_smem(bool sorted) {
        return build_keys(sorted) + sizeof(u16) * LS + (COMPACT ? 2 : 1) * sizeof(u16) * SPLATS;
    }
};

// Hash of a key: a sum of words times odd constants (linear, so that the hash of a neighbouring lattice point is
// the sum plus a constant, see link_neighbours), then a mix.
__host__ __device__ constexpr u64 hash_factor(int j) {
    u64 z = 0x9E3779B97F4A7C15ull * (u64)(j + 1);   // splitmix64 sequence
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (z ^ (z >> 31)) | 1ull;
}
template <int KW>
__device__ __forceinline__ u64 linear_hash(const Key<KW>& k) {
    u64 h = 0;
#pragma unroll
    for (int j = 0; j < KW; j++) h += k.w[j] * hash_factor(j);
    return h;
}
__device__ __forceinline__ u64 mix_hash(u64 h) {
    h ^= h >> 32;
    h *= 0xC4CEB9FE1A85EC53ull;
    return h ^ (h >> 29);
}
template <int KW>
__device__ __forceinline__ u64 hash_key(const Key<KW>& k) {
    return mix_hash(linear_hash<KW>(k));
}

template <int KW>
__device__ __forceinline__ bool key_equal(const Key<KW>& a, const Key<KW>& b) {
    bool eq = true;
#pragma unroll
    for (int j = 0; j < KW; j++) eq = eq && (a.w[j] == b.w[j]);
    return eq;
}

// Words that CTAs of one launch read, claim and write while others do: every such access is relaxed at GPU scope and of
// the whole word, since a narrower one beside a compare-and-swap of all of it would be a data race.
__device__ __forceinline__ u64 load_relaxed(const u64* p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_relaxed(u64* p, u64 v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void store_relaxed(u32* p, u32 v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// What a launch reads or writes once, and whose next reader comes after more than the caches hold, goes first when they need room, so that
// what is read again and again, value rows, keys and tables, stays: the point records (the construction's stores, the loads of splat and
// slice), the neighbours of a blur pass, the entries' keys and references beyond pd 5, new slots of the neighbour table.  us a call, plain / so:
// the records, 800x1200 x 3 167.3 / 165.2, 1024x1024 grey by RGB, forward + backward, 292 / 286, two volumes of 111x128x120 505 / 488, 8 x 512x512
// x 3
// 242 / 237; the neighbours 167.3 / 165.2, 291 / 286, five CRF steps on 375x500 x 21 381 / 374.5, 200 k points x 7 at pd 16 341 / 328 (beyond
// what stays in L2 see MOVED_ITEMS); the rest 164 / 165.2, 8 x 512x512 x 3 of noise 0.16 771 / 760, 1 M points with 16 features 1630 / 1613.
template <typename T>
__device__ __forceinline__ T load_once(const T* p) { return __ldcs(p); }
template <typename T>
__device__ __forceinline__ void store_once(T* p, T v) { __stcs(p, v); }
// A point's record.  Not up to pd 2, most calls of which are by position alone, where the items of a batch share one lattice's records (see
// one_for_all): 8 x 512x512 x 21 342 / 348.  Three to five dimensions may be positions alone too: 8 volumes of 64x64x64 x 21 181 / 185, but
// x 1 to 3 and four dimensions within 0.4 % of one another, and a choice at every load costs all calls 3 to 17 %.  Not beyond pd 5, where
// the compiler takes up to 16 registers more for it.
template <int PD, typename T>
__device__ __forceinline__ T load_record(const T* p) {
    if constexpr (PD > 2 && PD <= 5) return __ldcs(p);
    else return *p;
}

// load_once of a key: not for keys that this launch writes.
template <int KW>
__device__ __forceinline__ Key<KW> load_key_once(const Key<KW>* p) {
    Key<KW> k;
    const unsigned long long* w = reinterpret_cast<const unsigned long long*>(p);
#pragma unroll
    for (int j = 0; j < KW; j++) k.w[j] = load_once(w + j);
    return k;
}
// Key read straight from L2 (no L1): for data that another CTA of the SAME launch may have written.
template <int KW>
__device__ __forceinline__ Key<KW> load_key_l2(const Key<KW>* p) {
    Key<KW> k;
    const unsigned long long* w = reinterpret_cast<const unsigned long long*>(p);
#pragma unroll
    for (int j = 0; j < KW; j++) k.w[j] = __ldcg(w + j);
    return k;
}

// 16-bit field f of a key.  Fields 0..PD-1: lattice coordinates biased by 0x8000 (so that adding small
// offsets to a packed word never carries between fields); field PD: batch item.
template <int KW>
__device__ __forceinline__ void key_set(Key<KW>& k, int f, u16 v) {
    k.w[f >> 2] |= (u64)v << (16 * (f & 3));
}
template <int KW>
__device__ __forceinline__ u16 key_get(const Key<KW>& k, int f) {
    return (u16)(k.w[f >> 2] >> (16 * (f & 3)));
}

// 0x0001 in every coordinate field of key word j.
template <int PD>
__host__ __device__ constexpr u64 coord_ones(int j) {
    u64 m = 0;
    for (int f = 4 * j; f < 4 * j + 4; f++)
        if (f < PD) m |= 1ull << (16 * (f & 3));
    return m;
}

// Tile of this CTA.  Tile kernels run on a 3-D grid (tile column, tile row, item * outer + outer index)
// whenever that fits the grid limits, so no thread divides to find its tile; else on a 1-D grid.
struct TilePos {
    int tile, item, o, ty, tx;   // tile: whose records and range of entries these points have
};
__device__ __forceinline__ TilePos tile_at(const Geom& g, int x, int z) {   // CTA (x, blockIdx.y, z)
    TilePos t;
    if (g.grid3) {
        t.tx = x;
        t.ty = blockIdx.y;
        if (g.outer == 1) {
            t.item = z;
            t.o = 0;
        } else {
            t.item = z / g.outer;
            t.o = z - t.item * g.outer;
        }
        t.tile = ((g.lattice_items > 1 ? t.o : z) * g.tiles_y + t.ty) * g.tiles_x + t.tx;
    } else {
        t.tile = x;
        t.item = t.tile / g.tiles_per_item;
        int r = t.tile - t.item * g.tiles_per_item;
        if (g.lattice_items > 1) t.tile = r;
        const int per_plane = g.tiles_x * g.tiles_y;
        t.o = r / per_plane;
        r -= t.o * per_plane;
        t.ty = r / g.tiles_x;
        t.tx = r - t.ty * g.tiles_x;
    }
    return t;
}

// Where one lattice serves several items (see one_for_all), every item has its own value rows and its own copy of the list of
// entries, which names them, `item_entries` apart: what an item adds to its tiles' first entries.  (Added to the rows' address
// instead, it cost the splat of narrow rows up to 28 bytes of spills, and at pd 5 an SM's sixth CTA.)  A call by position alone has at most MAX_SDIMS
// feature dimensions.  (Without that said, slice_tiles_fast<16, 24> spilled 40 -> 104 bytes.)
template <int PD>
__device__ __forceinline__ int first_entry_of(const Geom& g, int item) {
    if constexpr (PD <= MAX_SDIMS) return item * (int)g.item_entries;
    else return 0;
}

__device__ __forceinline__ TilePos this_tile(const Geom& g) { return tile_at(g, blockIdx.x, blockIdx.z); }

// Point handled by thread `tid` of the tile: item, point index inside the item, validity; the long
// form also gives the point's position (outer index, row, column).
__device__ __forceinline__ bool tile_point(const Geom& g, const TilePos& t, int tid, int& item, int& pix, int& o,
                                           int& y, int& x) {
    item = t.item;
    o = t.o;
    const int ly = tid >> g.tx_log2, lx = tid & (g.TX - 1);
    y = t.ty * g.TY + ly;
    x = t.tx * g.TX + lx;
    pix = (o * g.H + y) * g.W + x;
    return (y < g.H) && (x < g.W);
}
__device__ __forceinline__ bool tile_point(const Geom& g, const TilePos& t, int tid, int& item, int& pix) {
    int o, y, x;
    return tile_point(g, t, tid, item, pix, o, y, x);
}

// Feature vector of a point.  Op path: src/PermutohedralLatticeCPU.h:464-473 (coordinate of each
// spatial dimension as float divided by spatial_std, reference channel divided by feature_std; IEEE
// divisions, not reciprocal multiplies).  The last two spatial coordinates are the point's row and
// column in its tile grid; only deeper dimensions need the reference's divide-and-modulo.
// Positions path: a row of the positions array.
template <int PD>
__device__ __forceinline__ void load_features(const Geom& g, const float* __restrict__ positions,
                                              const float* __restrict__ reference, int item, int pix, int o,
                                              int y, int x, float* f) {
    if (g.from_positions) {
        const float* p = positions + ((size_t)item * g.n + pix) * PD;
#pragma unroll
        for (int i = 0; i < PD; i++) f[i] = __ldg(p + i);
    } else {
        const float* ref = reference + ((size_t)item * g.n + pix) * g.R;
        int rest = o;
#pragma unroll
        for (int i = PD - 1; i >= 0; i--) {
            if (i >= g.n_sdims) {
                const float a = __ldg(ref + (i - g.n_sdims));
                f[i] = g.rcp_div ? div_by_rcp(a, g.feature_std, g.feature_rcp) : PL_FDIV(a, g.feature_std);
            } else {
                int c;
                if (i == g.n_sdims - 1 && g.n_sdims >= 2) {
                    c = x;
                } else if (i == g.n_sdims - 2) {
                    c = y;
                } else if (g.n_sdims == 1) {
                    c = x;
                } else {   // (what is left for the first dimension lies inside it: a volume's plane needs no division)
                    c = i ? rest % g.sdims[i] : rest;
                    if (i) rest /= g.sdims[i];
                }
                const float a = small_int_to_float(c);
                f[i] = g.rcp_div ? div_by_rcp(a, g.spatial_std, g.spatial_rcp) : PL_FDIV(a, g.spatial_std);
            }
        }
    }
}

// T = double: the reference's expressions as they stand (int converted to double, IEEE divisions).
template <int PD>
__device__ __forceinline__ void load_features(const Geom& g, const double* __restrict__ positions,
                                              const double* __restrict__ reference, int item, int pix, int o,
                                              int y, int x, double* f) {
    if (g.from_positions) {
        const double* p = positions + ((size_t)item * g.n + pix) * PD;
#pragma unroll
        for (int i = 0; i < PD; i++) f[i] = __ldg(p + i);
    } else {
        const double* ref = reference + ((size_t)item * g.n + pix) * g.R;
        int rest = o;
#pragma unroll
        for (int i = PD - 1; i >= 0; i--) {
            if (i >= g.n_sdims) {
                f[i] = __ddiv_rn(__ldg(ref + (i - g.n_sdims)), g.feature_std_d);
            } else {
                int c;
                if (i == g.n_sdims - 1 && g.n_sdims >= 2) {
                    c = x;
                } else if (i == g.n_sdims - 2) {
                    c = y;
                } else if (g.n_sdims == 1) {
                    c = x;
                } else {
                    c = i ? rest % g.sdims[i] : rest;
                    if (i) rest /= g.sdims[i];
                }
                f[i] = __ddiv_rn((double)c, g.spatial_std_d);
            }
        }
    }
}

// Floats of a vertex row: vd padded to a multiple of 4 (16-byte rows).
__host__ __device__ __forceinline__ int padded_vd(int vd) { return (vd + 3) & ~3; }

// Status word of the call, read once per CTA so that every thread takes the same branch even while
// other CTAs of the same launch are setting error bits.
__device__ __forceinline__ bool call_failed(const Header* hdr) {
    __shared__ u32 status_s;
    if (threadIdx.x == 0) status_s = hdr->status;
    __syncthreads();
    return status_s != 0;
}

// A call that failed on the device (status word set by an earlier launch) must not leave bytes that
// could pass for a result: the slice stage then fills the tile's output rows with NaN and returns.
template <typename T>
__device__ __forceinline__ void poison_tile_output(const Geom& g, T* __restrict__ output, int channels) {
    const TilePos tpos = this_tile(g);
    int item, pix;
    if (!tile_point(g, tpos, threadIdx.x, item, pix)) return;
    T* row = output + ((size_t)item * g.n + pix) * channels;
    const T nan = (T)__int_as_float(0x7FC00000);
    for (int j = 0; j < channels; j++) row[j] = nan;
}

// ---------------------------------------------------------------------------------------------
// Value rows.  A vertex row holds vd floats padded to VP = a multiple of 4, so that rows are 16-byte
// aligned: every row access below is a float4, and a row of 22 channels covers exactly three
// 32-byte sectors.  Pad channels stay zero through splat and blur and are never sliced.
// ---------------------------------------------------------------------------------------------
// Two floats an instruction, each rounded as by the scalar one.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<u64*>(&a)), "l"(*reinterpret_cast<u64*>(&b)), "l"(*reinterpret_cast<u64*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<u64*>(&a)), "l"(*reinterpret_cast<u64*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<u64*>(&a)), "l"(*reinterpret_cast<u64*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}

// Vector reduction into global memory (sm_90+): one L2 operation per 16 bytes.
__device__ __forceinline__ void red_add_v4(float* addr, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z),
                 "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ void red_add_v2(float* addr, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void red_add_f64(double* addr, double a) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(addr), "d"(a) : "memory");
}
__device__ __forceinline__ void red_add_f32(float* addr, float a) {
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(a) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// How a warp's lanes are spread over value rows: GS lanes (one float4 each) per row, PPW rows per
// warp instruction.  Rows wider than 32 quads are walked in chunks of 32 quads.
struct LaneMap {
    int gs, ppw, g, q0;
    bool active;
    __device__ __forceinline__ LaneMap(int qpr, int lane) {
        gs = qpr < 32 ? qpr : 32;
        ppw = 32 / gs;
        g = lane / gs;
        q0 = lane - g * gs;
        active = g < ppw;
    }
};

// ---------------------------------------------------------------------------------------------
// Bulk asynchronous copies (TMA engine, untiled form) with an mbarrier; every wait is bounded.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(u64* bar, unsigned count) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(u64* bar, unsigned bytes) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
// global -> shared, 16-byte aligned addresses, size a multiple of 16 bytes
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gmem_src, unsigned bytes, u64* bar) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(d),
                 "l"(gmem_src), "r"(bytes), "r"(a)
                 : "memory");
}
// Waits for phase `parity` of the barrier; gives up (returns false) after a bounded number of polls.
__device__ __forceinline__ bool mbar_wait(u64* bar, unsigned parity) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    for (int it = 0; it < (1 << 20); it++) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// shared -> global
__device__ __forceinline__ void bulk_store(void* gmem_dst, const void* smem_src, unsigned bytes) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem_src);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst), "r"(sa), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_store_finish() {
    asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void fence_async_proxy() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// A kernel launched with programmatic stream serialisation may become resident while the kernel before it in the
// stream is still draining: the first instruction waits until that kernel has finished and its writes are visible,
// the second lets the kernel AFTER this one become resident in its turn (its CTAs are scheduled once every CTA of
// this grid has got here).  First statement of most kernels; some wait later (the tile kernels, the blur passes, absmax_kernel) and until
// then read only what is older than the kernel before them (build_tiles also writes records, which no kernel of an earlier call still reads:
// clear_header is launched plainly), which holds since:
//   - no thread that releases has not waited, absmax_kernel aside, so that a kernel finds all finished but the one before it;
//   - absmax_kernel reads the call's input alone before it waits, and every CTA of it waits before it ends, so that it is finished after the
//     kernel before it.  That one is clear_header, launched plainly, or zero_rows, the first of an apply and overlapped with whoever wrote the
//     input: either has waited when absmax_kernel starts.
// The release comes after the wait on purpose: released first, a waiting kernel lets the one after it wait beside it, and
// two kernels' worth of waiting CTAs on the SMs slowed a long-running tile kernel by a quarter (pd = 16).
// Both instructions do nothing in a plain launch.
__device__ __forceinline__ void after_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// The first half alone, for kernels whose grid runs in several waves (the tile kernels) or whose CTAs all need their slots
// to the end (the inserts): they never release the next kernel, which then starts when the last of their CTAs has ended.
// Released at their start, the next kernel's CTAs sat on the SMs beside the tile kernel's later waves and slowed them (a
// call 15 % slower); released by every thread ahead of its last row, the splat still cost the dense CRF 16 x 512x512 x 21
// a tenth (forward + backward 1764 -> 1953 us).
__device__ __forceinline__ void wait_for_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The second half alone, for a kernel that starts on what is older than the kernel before it and waits for that at its end.
__device__ __forceinline__ void let_next_kernel_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// First point and number of valid points of tile row `ly` (the run of points that is contiguous in
// memory); returns false if the row lies outside the item.
__device__ __forceinline__ bool tile_row(const Geom& g, const TilePos& tpos, int ly, int& first_row, int& count) {
    int item, pix;
    if (!tile_point(g, tpos, ly * g.TX, item, pix)) return false;
    const int x0 = pix % g.W;
    first_row = item * g.n + pix;
    count = min(g.TX, g.W - x0);
    return true;
}

}  // namespace pl
