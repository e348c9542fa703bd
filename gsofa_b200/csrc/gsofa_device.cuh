// gsofa_device.cuh -- device code of the B200 symbolic factorization.
//
// Layout of one factorization job in HBM (all matrices of a batch share it):
//   per matrix  : n, line_base, G = (ptr[n+1], adj[]) and G^T = (ptr, adj),
//                 compact int32 CSR without diagonal entries;
//   per line l  : cnt[2][L] int32   -- |hi(s)| of pass 0 (U row) / 1 (L column)
//                 nxt[2][L] uint8   -- s+1 in hi(s)
//                 poff[2][L] int64  -- where the sorted hi(s) list sits in pool
//                 gptr[2][L+1] int64-- CSR offsets after compaction
//                 lrow[L] int32     -- |L row s| (histogram of the L columns)
//                 snind[L] uint8    -- line starts a supernode
//   pool / out  : int32 pattern entries (the traversals write pool, one range
//                 per chain of sources; compaction writes out in line order);
//   per traversal (two a CTA, one a pass, in the paired kernels):
//                 a frontier queue of qcap int32 (every vertex enters at most
//                 once per source, so qcap >= n never overflows);
//                 pattern mode: two rows of n uint16 stamps, the chain index at
//                 which each vertex was first set (one row is being written
//                 while the other's lists go out), and a chain's vertices
//                 (where memory is short: one row, the vertices in the queue);
//                 up to SNAP_MAX bitmaps of finished traversals (snapshots).
// The visited set is an n-bit bitmap with two summary levels, in shared memory
// or, for large n, in global memory.
//
// A traversal is led by one warp: it seeds each source, runs its small levels
// and decides what the source can reuse.  The other warps of its half of the
// CTA wait for work from it: large levels, clearing, lists, snapshots.
#pragma once

#include <cooperative_groups.h>
#include <stdint.h>

namespace gsofa {
namespace dev {

namespace cg = cooperative_groups;

// Rows of at most SLOT_NB ids are also kept whole in a 32-byte slot per
// vertex -- {degree, input degree, up to six ids} -- so expanding a frontier
// vertex is one L2 round trip instead of two (row bounds, then ids); longer
// rows' slots hold their offset instead and their ids are taken from adj.  Matrices whose mean
// off-diagonal degree is above SLOT_NB have no slots (slot == nullptr): most
// of their rows would pay the 32-byte slot load and still read adj.
constexpr int SLOT_NB = 6;

struct PassGraph {
    const int32_t *ptr;  // [n+1]
    const int32_t *adj;  // [ptr[n]]
    const int4 *slot;    // [2n + 2]: vertex v at slot[2v], slot[2v+1], then an empty slot (or null)
};

struct MatDesc {
    int32_t n;
    int32_t pad;
    int64_t line_base;   // first line of this matrix in the job's line space
    PassGraph g[2];      // 0: G, 1: G^T
    const int32_t *rawdeg; // [n] input degree of every line (work counters)
};

// The sources of one matrix, s = offset + stride * j for j in [0, nj), cut
// into pieces of consecutive j.  Piece k of a range covers pass k & 1 (one
// pass per piece unless paired) and piece k >> 1 (k, paired) counted from the
// top: the highest sources, which carry the largest traversals, are handed
// out first.  The top nj - tail sources go in pieces of `chunk`, the bottom
// `tail` ones in pieces of `small`, handed out last, so a launch ends on
// short pieces instead of waiting for a long one.
struct Range {
    int32_t mat;
    int32_t chunk;
    int32_t nj;
    int32_t stride;
    int32_t offset;
    int32_t small;       // piece length of the bottom `tail` sources
    int32_t tail;
    int32_t pad;
    int64_t piece_base;  // first global piece index of this range
    int64_t npieces;     // pieces of both passes
};

// Sources [j0, j1) of piece c of a range, counted from its top.
__host__ __device__ inline void piece_bounds(const Range &rg, int64_t c, int64_t &j0, int64_t &j1)
{
    const int64_t top = (int64_t)rg.nj - rg.tail;
    const int64_t nb = (top + rg.chunk - 1) / rg.chunk;
    if (c < nb) {
        j1 = (int64_t)rg.nj - c * rg.chunk;
        j0 = j1 - rg.chunk > (int64_t)rg.tail ? j1 - rg.chunk : (int64_t)rg.tail;
    } else {
        j1 = (int64_t)rg.tail - (c - nb) * rg.small;
        j0 = j1 - rg.small > 0 ? j1 - rg.small : 0;
    }
}

// Pieces of one pass of a range.
__host__ __device__ inline int64_t pieces_per_pass(const Range &rg)
{
    const int64_t top = (int64_t)rg.nj - rg.tail;
    return (top + rg.chunk - 1) / rg.chunk + ((int64_t)rg.tail + rg.small - 1) / rg.small;
}

// Shared pieces (paired passes with reuse, automatic piece length).  A CTA's
// piece is a stretch of units of 8 sources of one range, which it claims from
// below, an eighth of what is left at a time, while CTAs that have run out of
// pieces take its upper part: a word per CTA holds {range, end, next unit}, and
// a second one the costliest step so far beyond an average unit (a traversal
// from nothing, which whoever takes a part has to run) and an average unit, in
// 256 cycles.
constexpr int UNIT = 8;
constexpr int CLAIM_MAX = 8;   // units claimed at a time
constexpr int UNIT_BITS = 20;
constexpr unsigned long long UNIT_MASK = (1ull << UNIT_BITS) - 1;

__device__ __forceinline__ unsigned long long piece_word(int range, int end, int next)
{
    return (unsigned long long)range << (2 * UNIT_BITS) | (unsigned long long)end << UNIT_BITS |
           (unsigned long long)next;
}

// Error bits reported through JobArgs::status.
enum : uint32_t {
    ERR_POOL_OVERFLOW = 1u,
    ERR_COUNT_MISMATCH = 4u,   // a list's running count and its bitmap disagree
};

struct JobArgs {
    const MatDesc *mats;
    int32_t nmats;
    int32_t nranges;
    const Range *ranges;
    int64_t npieces;
    unsigned long long *piece_counter; // dynamic fetch of work pieces
    unsigned long long *shared_piece;  // shared pieces: a word per CTA (or null)
    unsigned long long *shared_cost;   // ... and what its sources cost
    unsigned *fresh_cost;      // ... and the first claims of pieces, by where they begin
    int32_t *queue;            // gridDim.x * qcap
    int64_t qcap;
    int32_t bitmap_words;      // shared-memory bitmap size (>= max n / 32, multiple of 128)
    int32_t state_words;       // STATE_PAD, bitmap, its two summary levels
    int32_t ring_size;         // shared-memory frontier ring entries (power of two)
    int32_t snap_k;            // snapshots a traversal slot keeps (0: none)
    int32_t reuse;
    int32_t want_pattern;
    int32_t max_sn;
    int64_t L;                 // total lines
    int32_t *cnt;              // [2][L]
    uint8_t *nxt;              // [2][L]
    int64_t *poff;             // [2][L]
    int32_t *pool;
    int64_t pool_cap;
    unsigned long long *pool_tail;
    int64_t *gptr;             // [2][L+1]
    int32_t *out;              // pool_cap entries
    int32_t *lrow;             // [L]
    uint8_t *snind;            // [L]
    int32_t *sn_list;          // [L]
    int64_t *mat_info;         // [nmats][3] at each matrix's first line: pass-0 and
                               // pass-1 CSR offsets, supernodes before it
    int64_t ntiles;
    int64_t tile_lo, tile_hi;  // the post-traversal phases cover tiles [tile_lo, tile_hi)
                               // (all of them, unless only a line range was processed)
    int64_t *tile_sum;         // [2][ntiles] then exclusive prefix (in place)
    int64_t *tile_last;        // [ntiles] last supernode-run start, then prefix max
    int64_t *tile_sn;          // [ntiles] then exclusive prefix
    unsigned long long *counters; // [0] edges inspected, [1] sources, [2] sn total,
                                  // [3] pass-G expansions, [4] pass-G input degrees,
                                  // [5] levels, [6] sources that reused state,
                                  // [7..13] cycles: the sources' own steps, their
                                  // levels, snapshots, (unused), list output,
                                  // clearing, pair wait;
                                  // [14] ns until the traversals ended,
                                  // [15] CTAs' traversal ns, summed
    uint32_t *status;
    uint16_t *stamp;           // pattern mode: per traversal, two rows of stamp_stride
    int64_t stamp_stride;      // entries: the chain index at which each vertex was first set
    int64_t stamp_other;       // entries from a traversal's first row to its other one; 0: it has
                               // one row, and no work goes on beside its list output
    int32_t *lists;            // pattern mode: qcap entries per traversal (its queue, with one row)
    uint32_t *snap;            // snapshots: snap_k bitmaps per traversal slot
    uint32_t *gbm;             // global-state kernels: per traversal, state_words
                               // words (bitmap and its summaries) in global memory
    unsigned int *blk_done;    // ranges form, streamed: entries written into each
    int32_t blk_shift;         // pool block of 2^blk_shift entries (or null)
};

constexpr int TILE = 2048;     // lines per tile in the post-traversal phases

__device__ __forceinline__ int64_t warp_incl_scan(int64_t x)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Exclusive scan over the block; *total receives the block sum.  Uses
// s_warp[32]; contains two __syncthreads and a trailing one.
template <int BLOCK>
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t *total,
                                                   int64_t *s_warp)
{
    constexpr int NW = BLOCK / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t x = warp_incl_scan(v);
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int64_t w = lane < NW ? s_warp[lane] : 0;
        w = warp_incl_scan(w);
        if (lane < NW) s_warp[lane] = w;
    }
    __syncthreads();
    int64_t pre = wid ? s_warp[wid - 1] : 0;
    *total = s_warp[NW - 1];
    __syncthreads();
    return pre + x - v;
}

template <int BLOCK>
__device__ __forceinline__ int64_t block_sum(int64_t v, int64_t *s_warp)
{
    int64_t t;
    block_excl_scan<BLOCK>(v, &t, s_warp);
    return t;
}

// Exclusive max-scan over the block (identity -1); *total receives the
// block maximum.
template <int BLOCK>
__device__ __forceinline__ int64_t block_excl_max(int64_t v, int64_t *total,
                                                  int64_t *s_warp)
{
    constexpr int NW = BLOCK / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = max(x, y);
    }
    int64_t ex = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) ex = -1;
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int64_t w = lane < NW ? s_warp[lane] : -1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w = max(w, y);
        }
        if (lane < NW) s_warp[lane] = w;
    }
    __syncthreads();
    int64_t pre = wid ? s_warp[wid - 1] : -1;
    *total = s_warp[NW - 1];
    __syncthreads();
    return max(pre, ex);
}

// Global load; CG = true reads through L2 only (no L1), for data that the
// host may rewrite while a persistent kernel runs.
template <bool CG>
__device__ __forceinline__ int32_t ld(const int32_t *p)
{
    if (CG) return __ldcg(p);
    return *p;
}

template <bool CG>
__device__ __forceinline__ int4 ld4(const int4 *p)
{
    if (CG) return __ldcg(p);
    return *p;
}

// Words of ones before a traversal's bitmap (a 16-byte group; id -1 has the last).
constexpr int STATE_PAD = 4;

// The visited set of one traversal: a bitmap of `words` words (a multiple of
// 128) followed by its summaries, one bit per bitmap word and then one bit per
// summary word (per 32K vertices), so that output, clearing and copying skip
// empty stretches.  Words are numbered through all three.  A summary bit is
// only ever added while a state grows, so neither level is read back then.
//
// In shared memory the words are addressed in the shared window (one register,
// and no generic loads or atomics whatever the code around them).
template <bool GBM>
struct Bits;

template <>
struct Bits<false> {
    uint32_t base;   // shared-window address
    int words;
    __device__ __forceinline__ uint32_t get(int i) const
    {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(base + 4u * (uint32_t)i));
        return v;
    }
    __device__ __forceinline__ uint4 get4(int i4) const
    {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(base + 16u * (uint32_t)i4));
        return v;
    }
    __device__ __forceinline__ void put(int i, uint32_t v) const
    {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + 4u * (uint32_t)i), "r"(v) : "memory");
    }
    __device__ __forceinline__ void put4(int i4, uint4 v) const
    {
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(base + 16u * (uint32_t)i4), "r"(v.x), "r"(v.y),
                     "r"(v.z), "r"(v.w)
                     : "memory");
    }
    // Where vertex m's word is; m = -1 (no vertex) has the word before the
    // first, which is all ones.
    typedef uint32_t Place;
    __device__ __forceinline__ Place place(int32_t m) const { return base + (uint32_t)((m >> 3) & ~3); }
    __device__ __forceinline__ uint32_t peek(Place at, int32_t) const
    {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
        return v;
    }
    // Adds `bit` where it is not in w; w becomes the word as it was.
    __device__ __forceinline__ void add(Place at, uint32_t bit, uint32_t &w) const
    {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b32 x;\n\tand.b32 x, %0, %2;\n\tsetp.eq.u32 p, x, 0;\n\t"
            "@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
            : "+r"(w)
            : "r"(at), "r"(bit));
    }
    __device__ __forceinline__ void add_or(int i, uint32_t m, bool on) const
    {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.shared.or.b32 [%0], %1;\n\t}" ::"r"(
                         base + 4u * (uint32_t)i),
                     "r"(m), "r"((uint32_t)on));
    }
};

// In global memory (resident in L2 at the sizes that matter) the words change
// by atomics in L2 and are cleared by plain stores, so they are read through
// L2 only: an L1 copy could be stale.
template <>
struct Bits<true> {
    uint32_t *base;
    int words;
    __device__ __forceinline__ uint32_t get(int i) const { return __ldcg(base + i); }
    __device__ __forceinline__ uint4 get4(int i4) const { return __ldcg(reinterpret_cast<const uint4 *>(base) + i4); }
    __device__ __forceinline__ void put(int i, uint32_t v) const { base[i] = v; }
    __device__ __forceinline__ void put4(int i4, uint4 v) const { reinterpret_cast<uint4 *>(base)[i4] = v; }
    // A read before the atomic would cost as much as the atomic itself: `peek`
    // only tells vertices from -1.
    typedef int Place;
    __device__ __forceinline__ Place place(int32_t m) const { return m >> 5; }
    __device__ __forceinline__ uint32_t peek(Place, int32_t m) const { return m < 0 ? ~0u : 0u; }
    __device__ __forceinline__ void add(Place at, uint32_t bit, uint32_t &w) const
    {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b32 x;\n\tand.b32 x, %0, %2;\n\tsetp.eq.u32 p, x, 0;\n\t"
            "@p atom.relaxed.gpu.global.or.b32 %0, [%1], %2;\n\t}"
            : "+r"(w)
            : "l"(base + at), "r"(bit)
            : "memory");
    }
    __device__ __forceinline__ void add_or(int i, uint32_t m, bool on) const
    {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.relaxed.gpu.global.or.b32 [%0], %1;\n\t}" ::"l"(base + i),
            "r"(m), "r"((uint32_t)on)
            : "memory");
    }
};

template <bool GBM>
__device__ __forceinline__ Bits<GBM> bits_at(uint32_t *p, int words)
{
    if constexpr (GBM) return Bits<GBM>{p, words};
    else return Bits<GBM>{(uint32_t)__cvta_generic_to_shared(p), words};
}

// First words of the two summary levels, and the second one's length.
template <bool GBM>
__device__ __forceinline__ int summ1(const Bits<GBM> &b) { return b.words; }
template <bool GBM>
__device__ __forceinline__ int summ2(const Bits<GBM> &b) { return b.words + (b.words >> 5); }
template <bool GBM>
__device__ __forceinline__ int summ2_words(const Bits<GBM> &b) { return ((b.words >> 5) + 31) >> 5; }

// Enters bitmap word wi, which just became nonzero, in both summary levels.
template <bool GBM>
__device__ __forceinline__ void mark_word(const Bits<GBM> &b, int wi, bool on)
{
    b.add_or(summ1(b) + (wi >> 5), 1u << (wi & 31), on);
    b.add_or(summ2(b) + (wi >> 10), 1u << ((wi >> 5) & 31), on);
}

// Frontier queue of one source: absolute positions 0, 1, 2, ... in BFS order.
// A position p written while the writer's level started at w0 lives in the
// shared-memory ring (a power of two of entries) when p - w0 < ring_size and in
// the traversal's global spill array otherwise; readers apply the same rule
// with the same w0.  Ring entries of one level and of the level it feeds always
// lie within ring_size consecutive positions, so live ring slots never collide.
// A vertex enters at most once per source, so positions stay below n.
struct Frontier {
    uint32_t ring;    // shared-window address
    int ring_size;
};

// Queues m at p where the bit was not in w and m < s.
__device__ __forceinline__ void ring_put(const Frontier &f, int p, int32_t m, uint32_t w, uint32_t bit, int32_t s)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b32 x;\n\tand.b32 x, %2, %3;\n\tsetp.eq.u32 p, x, 0;\n\t"
        "setp.lt.and.s32 q, %1, %4, p;\n\t@q st.shared.u32 [%0], %1;\n\t}" ::"r"(
            f.ring + 4u * (uint32_t)(p & (f.ring_size - 1))),
        "r"(m), "r"(w), "r"(bit), "r"(s));
}

__device__ __forceinline__ void spill_put(int32_t *at, int32_t m, uint32_t w, uint32_t bit, int32_t s)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b32 x;\n\tand.b32 x, %2, %3;\n\tsetp.eq.u32 p, x, 0;\n\t"
        "setp.lt.and.s32 q, %1, %4, p;\n\t@q st.global.u32 [%0], %1;\n\t}" ::"l"(at),
        "r"(m), "r"(w), "r"(bit), "r"(s)
        : "memory");
}

__device__ __forceinline__ int32_t ring_get(const Frontier &f, int p)
{
    int32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(f.ring + 4u * (uint32_t)(p & (f.ring_size - 1))));
    return v;
}

__device__ __forceinline__ void fr_put(const Frontier &f, int32_t *spill, int p, int w0, int32_t m, bool on)
{
    const bool in = p - w0 < f.ring_size;
    ring_put(f, p, m, on && in ? 0u : 1u, 1u, INT32_MAX);
    if (on && !in) spill[p] = m;
}

// The ring's entry at p where p < end, else `none`.
__device__ __forceinline__ int32_t ring_get(const Frontier &f, int p, int end, int32_t none)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p ld.shared.u32 %0, [%1];\n\t}"
                 : "+r"(none)
                 : "r"(f.ring + 4u * (uint32_t)(p & (f.ring_size - 1))), "r"(p), "r"(end));
    return none;
}

__device__ __forceinline__ int32_t fr_get(const Frontier &f, const int32_t *spill, int p, int w0)
{
    return p - w0 < f.ring_size ? ring_get(f, p) : spill[p];
}

// Seeding window: the rows of up to SEED_WIN consecutive sources (SEED_ADJ
// ids at most), loaded together -- consecutive rows are one stretch of the
// adjacency array -- so a source's seeding reads shared memory instead of
// waiting on two dependent L2 round trips.
constexpr int SEED_WIN = 32;
constexpr int SEED_ADJ = 512;

// Snapshots of finished traversals (paired passes): at most SNAP_MAX a
// traversal slot, each usable by the sources of the SNAP_REACH words of lines
// from its own source on.
constexpr int SNAP_MAX = 8;
constexpr int SNAP_REACH = 16;

// Levels of at most this many vertices are run by a traversal's leader alone.
constexpr int SOLO_MAX = 16;

// Work that a traversal's first warp (its leader) hands to its other warps, the
// helpers.
enum : int { OP_EXIT = 0, OP_LEVELS, OP_CLEAR, OP_LISTS, OP_SAVE, OP_MERGE };

// A CTA's shared piece (word == nullptr: the piece is the CTA's alone).
struct SharedPiece {
    unsigned long long *word, *cost;
    int32_t first, last;   // the range's sources [first, last)
    int32_t s_lo;          // the piece's first source
    volatile unsigned *fresh;   // where the cost of its first claim goes (JobArgs::fresh_cost)
};

// What a traversal needs now and then: kept in shared memory, since the
// leader's registers are short.
struct Home {
    PassGraph g;             // the piece's pass graph
    const int32_t *rawdeg;   // and input degrees
    int32_t *spill;          // the frontier's entries past the ring
    uint16_t *stamps;        // pattern mode: two stamp rows
    int32_t *lists;          // pattern mode: a chain's vertices while its lists are written
    uint32_t *snaps;         // snapshots
    int64_t row;             // cnt / nxt / poff entry of the matrix's line 0 in this pass
    int32_t *lrow;           // L row counts of the matrix's lines (pass G^T), or null
    int32_t n;
    int32_t pass;
};

// One traversal's shared state.  The leader warp runs the piece's sources and
// alone touches the fields marked L; the other warps wait at the traversal's
// barrier for an op, and the fields marked O are its arguments and results.
struct SharedState {
    Home home;
    int op;                 // O: OP_*
    int src, cidx;          // O: the source, its index in its chain
    int lv_start, lv_end, lv_wstart;   // O: OP_LEVELS: the level to start from
    int snap, lo, hi, t;    // O: OP_SAVE / OP_MERGE: slot, its bitmap words, its source
    int tailc[3];           // level entry counts by phase
    int run_cut[2];         // by exchange: sources of the pass's next run, and of its window << 8
    int fetch[3];           // dynamic fetch counters by phase
    int nh;                 // O: new vertices above the source that an op found
    int npush;              // O: queue entries that OP_MERGE made
    int seg[2];             // piece boundaries after chain alignment
    SharedPiece own;        // (the first traversal's) the CTA's piece
    volatile int next_end;  // shared pieces: where the claimed sources end
    unsigned long long claim;   // ... the piece's word at the last claim
    int claimed;            // ... units claimed there
    int unit_done;          // ... sources done when it was made
    unsigned unit_t, unit_sum, unit_mean, unit_most;   // ... when, what all units but the first took, a unit
                            // takes on average, and the costliest step beyond that, in 256 cycles
    // list output (pattern mode): the chain -- consecutive sources sharing one
    // bitmap -- whose lists are written when it ends
    uint16_t *stamp;        // the chain's stamp row, or null (counts only)
    int chain_s0;           // its first source
    int chain_first, chain_len;   // the lists to write: those of its sources [first, len)
    int chain_hi;           // no vertex above is set
    int64_t chain_total;    // entries of those lists
    int64_t warp[32];       // per-warp counts of a chain's vertices
    long long pool_base;    // the chain's pool range (-1: pool short)
    // tallies, kept by the leader's first lane: levels, then cycles of the
    // sources' own steps, their levels, list output, clearing, snapshots, wait
    // for the other pass; sources; those that started afresh
    unsigned long long prof[8];
    unsigned long long nsrc, nfresh;
    unsigned long long work[3];   // edges, pass-G expansions, pass-G input degrees
    uint32_t carry[3];            // ... and 2^31s of them
    int snaps;              // L: snapshots taken in this piece
    int snap_credit;        // L: what traversals and snapshots taken over have earned, in vertices (-1: none yet)
    int weight;             // L: vertices queued by the state's traversals
    uint32_t reach[2][SNAP_REACH];            // by exchange: this bitmap's words from the source's on
    uint32_t snap_reach[SNAP_MAX][SNAP_REACH];  // L: the other pass's words when the snapshot was taken
    int snap_t[SNAP_MAX], snap_lo[SNAP_MAX], snap_hi[SNAP_MAX], snap_w[SNAP_MAX];   // L: source (-1: empty),
                                              // words, vertices its traversals queued
    int32_t win_adj[SEED_ADJ];                // L: the window's rows
    int32_t ev_x[33], ev_p[33];               // L: a run's new ids and their places in the window
};

__device__ __forceinline__ void init_state(SharedState &sh)
{
    sh.stamp = nullptr;
    sh.nh = 0;
    for (int q = 0; q < 8; q++) sh.prof[q] = 0;
    sh.nsrc = sh.nfresh = 0;
    sh.work[0] = sh.work[1] = sh.work[2] = 0;
    sh.carry[0] = sh.carry[1] = sh.carry[2] = 0;
    sh.tailc[0] = sh.tailc[1] = sh.tailc[2] = 0;
    sh.fetch[0] = sh.fetch[1] = sh.fetch[2] = 0;
}

// A traversal's home moves to pass `pass` of a matrix (its leader's first lane).
__device__ __forceinline__ void settle(Home &h, const JobArgs &a, const MatDesc &md, int pass)
{
    h.g = md.g[pass];
    h.rawdeg = md.rawdeg;
    h.row = (int64_t)pass * a.L + md.line_base;
    h.lrow = pass && a.want_pattern ? a.lrow + md.line_base : nullptr;
    h.n = md.n;
    h.pass = pass;
}

// A CTA's shared memory begins with this; bitmaps and rings follow.  It is at
// the beginning of the dynamic part so that functions that are not inlined
// reach it by a known shared address: the leader's and the helpers' code are
// functions of their own, whose registers are allocated apart (as one body they
// came out 20% slower or faster with every unrelated change).
template <int NS, int HISTS>
struct Cta {
    JobArgs a;
    SharedState t[NS];
    volatile int pair_flag[2][2];   // [exchange parity][pass]: s+1 in hi(s), or a run's set sources
    volatile long long piece;
    volatile unsigned long long word;
    int hist[HISTS][32];            // list output: a row a helper warp
};

template <int BLOCK, bool PAIRED, bool LISTS>
using CtaOf = Cta<PAIRED ? 2 : 1, LISTS ? (PAIRED ? BLOCK / 32 - 2 : BLOCK / 32 - 1) : 1>;

template <class C>
__device__ __forceinline__ C &cta()
{
    extern __shared__ __align__(16) uint32_t smem_dyn[];
    return *reinterpret_cast<C *>(smem_dyn);
}

// Bytes before the bitmaps (a multiple of 16).
__host__ __device__ constexpr size_t cta_bytes(int ns, int hists)
{
    return ((ns == 2 ? sizeof(Cta<2, 1>) : sizeof(Cta<1, 1>)) + (size_t)(hists - 1) * 128 + 15) / 16 * 16;
}

// Barrier of the GT threads that work on one traversal: the whole CTA or one
// half of it, through the named barrier `bar` (1 or 2).
template <int GT>
__device__ __forceinline__ void gsync(int bar)
{
    if (bar == 1) asm volatile("bar.sync 1, %0;" ::"n"(GT) : "memory");
    else asm volatile("bar.sync 2, %0;" ::"n"(GT) : "memory");
}

// Barrier of a traversal's helper warps (all but its leader).
template <int GT>
__device__ __forceinline__ void helper_sync(int bar)
{
    if (GT == 64) __syncwarp();
    else if (bar == 1) asm volatile("bar.sync 4, %0;" ::"n"(GT - 32) : "memory");
    else asm volatile("bar.sync 5, %0;" ::"n"(GT - 32) : "memory");
}

__device__ __forceinline__ uint32_t clock32()
{
    uint32_t c;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
    return c;
}

// Since c0 (clock32), in 256s of cycles: right on average, for steps of up to
// 2^32 cycles and sums of minutes.
__device__ __forceinline__ uint32_t since(uint32_t c0) { return ((clock32() >> 8) - (c0 >> 8)) & 0xffffffu; }

// Barrier of the two leader warps of a CTA that runs both passes of a source.
__device__ __forceinline__ void pair_sync()
{
    __syncwarp();
    asm volatile("bar.sync 3, 64;" ::: "memory");
}

// Visits the nonzero chunks c in [c0, c1) (chunk = 32 bitmap words = one
// summary word) in increasing order, using the second summary level to skip
// empty stretches; fn(c) runs warp-uniformly.
template <bool GBM, class F>
__device__ __forceinline__ void for_nonzero_chunks(const Bits<GBM> &b, int c0, int c1, F fn)
{
    int c = c0;
    while (c < c1) {
        const int wb = c & ~31;
        uint32_t m = b.get(summ2(b) + (wb >> 5)) & (~0u << (c & 31));
        if (c1 - wb < 32) m &= (1u << (c1 - wb)) - 1u;
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1u;
            fn(wb + k);
        }
        c = wb + 32;
    }
}

// True when x-1 is in adj(x); evaluated by one whole warp.
__device__ __forceinline__ bool warp_has_prev(const PassGraph &g, int32_t x)
{
    const int lane = threadIdx.x & 31;
    bool hit = false;
    for (int32_t k = g.ptr[x] + lane; k < g.ptr[x + 1]; k += 32)
        hit |= (g.adj[k] == x - 1);
    return __any_sync(0xffffffffu, hit);
}

// The chain start at or below x: the lowest y with y+1 .. x each holding its
// predecessor, searched at most `limit - 1` steps down; x itself when the
// chain reaches further (then the cut is not aligned).  One warp.
__device__ __forceinline__ int32_t chain_start(const PassGraph &g, int32_t x, int32_t limit)
{
    int32_t y = x;
    for (int step = 0; step < limit - 1; step++) {
        if (y == 0 || !warp_has_prev(g, y)) return y;
        y--;
    }
    return (y == 0 || !warp_has_prev(g, y)) ? y : x;
}

// What every warp of a traversal has in registers.
template <bool GBM>
struct Trav {
    Bits<GBM> bits;
    Frontier f;
    uint16_t *stamp;       // the chain's stamps (pattern mode, else null)
};

// Per-thread tallies of one work piece (folded into SharedState::work when it
// ends); the per-source ones live in SharedState, kept by one thread.
struct Tally {
    uint32_t edges = 0, xcnt = 0, einsp = 0;
    uint32_t slot = 0;   // sums of slot words: lanes 0, 8, .. degrees, lanes 1, 9, .. input degrees
};

// Before a traversal, which adds less than 2^31 to any tally (it expands a
// vertex once, and the input has less than 2^31 entries): 2^31 of each that has
// them move to SharedState::carry.
__device__ __forceinline__ void carry(SharedState &sh, Tally &acc, int lane)
{
    const uint32_t slot = (lane & 7) < 2 ? acc.slot : 0u;
    if ((int)(acc.edges | acc.xcnt | acc.einsp | slot) < 0) {
        const bool first = sh.home.pass == 0;   // the other pass counts edges only
        if ((int)acc.edges < 0) atomicAdd(&sh.carry[0], 1u);
        if ((int)acc.xcnt < 0 && first) atomicAdd(&sh.carry[1], 1u);
        if ((int)acc.einsp < 0 && first) atomicAdd(&sh.carry[2], 1u);
        if ((int)slot < 0 && ((lane & 7) == 0 || first)) atomicAdd(&sh.carry[(lane & 7) ? 2 : 0], 1u);
        acc.edges &= 0x7fffffffu;
        acc.xcnt &= 0x7fffffffu;
        acc.einsp &= 0x7fffffffu;
        acc.slot &= 0x7fffffffu;
    }
}

// The sum of a 32-bit tally over a warp, and its addition to a 64-bit counter.
__device__ __forceinline__ void fold_tally(unsigned long long *to, uint32_t v, int lane)
{
    const unsigned long long lo = __reduce_add_sync(0xffffffffu, v & 0xffffu);
    const unsigned long long hi = __reduce_add_sync(0xffffffffu, v >> 16);
    if (lane == 0) atomicAdd(to, lo + (hi << 16));
}

__device__ __forceinline__ void fold_work(SharedState &sh, Tally acc, int pass, int lane)
{
    carry(sh, acc, lane);
    __syncwarp();
    fold_tally(&sh.work[0], acc.edges + ((lane & 7) == 0 ? acc.slot : 0u), lane);
    if (pass) return;
    fold_tally(&sh.work[1], acc.xcnt, lane);
    fold_tally(&sh.work[2], acc.einsp + ((lane & 7) == 1 ? acc.slot : 0u), lane);
}

// One warp step: sets the bits m, one per lane and u (-1: none), all of them in
// flight together and without branches -- the words' reads first (not in global
// memory), then the atomics of those that look unset, then the summaries of
// words that became nonzero.  New vertices below s are queued for the next
// level (alloc(k) hands out k positions, warp-uniformly; w0 is the first
// position of the level whose vertices found them); the others, s itself
// included, are counted (the return value, warp-uniform).  Every new vertex
// above the chain's first source gets the chain index of s as its stamp
// (pattern mode).  The integer pipe bounds this code (it issues every other
// cycle, and ran at 80% of that on the 300 x 300 grid), so every instruction
// here is counted: predicates are formed inside the memory operations, and a
// lane without an id needs no test of its own.
template <int U, bool GBM, class Alloc>
__device__ __forceinline__ int visit(const Trav<GBM> &t, const SharedState &sh, const int32_t (&m)[U], int32_t s, int cidx, int w0,
                                     Alloc alloc)
{
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    uint32_t w[U], bit[U];
    typename Bits<GBM>::Place at[U];
    bool any = false;
#pragma unroll
    for (int u = 0; u < U; u++) {
        bit[u] = 1u << (m[u] & 31);
        at[u] = t.bits.place(m[u]);
        w[u] = t.bits.peek(at[u], m[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) any |= !(w[u] & bit[u]);
    if (!__any_sync(0xffffffffu, any)) return 0;
#pragma unroll
    for (int u = 0; u < U; u++) t.bits.add(at[u], bit[u], w[u]);
    any = false;
#pragma unroll
    for (int u = 0; u < U; u++) any |= w[u] == 0u;
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int u = 0; u < U; u++) mark_word(t.bits, m[u] >> 5, w[u] == 0u);
    }
    if (t.stamp != nullptr) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (!(w[u] & bit[u]) && m[u] > s - cidx) t.stamp[m[u]] = (uint16_t)cidx;
    }
    unsigned low[U];
    int nlow = 0, nhigh = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        low[u] = __ballot_sync(0xffffffffu, !(w[u] & bit[u]) && m[u] < s);
        nlow += __popc(low[u]);
        nhigh += __popc(__ballot_sync(0xffffffffu, !(w[u] & bit[u]) && m[u] >= s));
    }
    if (nlow) {
        int pos = alloc(nlow);
        if (pos + nlow - w0 <= t.f.ring_size) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                ring_put(t.f, pos + __popc(low[u] & below), m[u], w[u], bit[u], s);
                pos += __popc(low[u]);
            }
        } else if (pos - w0 >= t.f.ring_size) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                spill_put(sh.home.spill + pos + __popc(low[u] & below), m[u], w[u], bit[u], s);
                pos += __popc(low[u]);
            }
        } else {
#pragma unroll 1
            for (int u = 0; u < U; u++) {
                int32_t mu = m[0], lu = low[0];
#pragma unroll
                for (int k = 1; k < U; k++)
                    if (u == k) { mu = m[k]; lu = low[k]; }
                fr_put(t.f, sh.home.spill, pos + __popc(lu & below), w0, mu, (lu >> (threadIdx.x & 31)) & 1u);
                pos += __popc(lu);
            }
        }
    }
    return nhigh;
}

// The rows of up to 32 frontier vertices -- each lane holds the bounds of one,
// d ids from adj[b] on, or d = 0 -- edge by edge: the lanes share the rows' ids
// by a prefix sum of their lengths, so a warp's loads touch the rows' own
// sectors once.  (One lane per row, eight ids at a time, fetched a sector per
// id -- 32 rows' lines do not stay in the L1 that the bitmaps leave -- and ran
// the 200,003-line power-law counts at 0.31 edges per SM cycle.)
template <bool CG, bool GBM, class Alloc>
__device__ __forceinline__ int expand_edges(const Trav<GBM> &t, const SharedState &sh, int32_t b, int32_t d, int32_t s, int cidx, int w0,
                                            Alloc alloc)
{
    const int lane = threadIdx.x & 31;
    const unsigned upto = ~0u >> (31 - lane);   // lanes 0 .. lane
    int nh = 0;
    // the rows with ids first
    const unsigned some = __ballot_sync(0xffffffffu, d > 0);
    const int rows = __popc(some);
    if (some & (some + 1u)) {
        int from = 0;   // the lane of row `lane`: as many rows before it (a search; __fns is a loop)
#pragma unroll
        for (int o = 16; o; o >>= 1)
            if (__popc(some & ((1u << (from + o)) - 1u)) <= lane) from += o;
        b = __shfl_sync(0xffffffffu, b, from);
        d = __shfl_sync(0xffffffffu, d, from);
        if (lane >= rows) d = 0;
    }
    int incl = d;   // distinct vertices: their rows hold at most nnz < 2^31 ids together
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int excl = lane < rows ? incl - d : INT32_MAX;   // where row `lane` begins among the warp's ids
    const int32_t from = b - excl;                         // id e is adj[from + e] of its row
    // ids e0 .. e0 + 31, one a lane: a lane's row is the last one that begins
    // at or before its id
    auto id = [&](int e0) {
        const int before = __popc(__ballot_sync(0xffffffffu, excl < e0));
        const unsigned begins =
            __reduce_or_sync(0xffffffffu, (unsigned)(excl - e0) < 32u ? 1u << (excl - e0) : 0u);
        const int row = before + __popc(begins & upto) - 1;
        const int32_t at = __shfl_sync(0xffffffffu, from, row & 31) + e0 + lane;
        return e0 + lane < total ? ld<CG>(sh.home.g.adj + at) : -1;
    };
    int e0 = 0;
    for (; total - e0 > 32; e0 += 128) {   // 128 ids in flight
        int32_t m[4];
#pragma unroll
        for (int u = 0; u < 4; u++) m[u] = id(e0 + 32 * u);
        nh += visit<4, GBM>(t, sh, m, s, cidx, w0, alloc);
    }
    if (e0 < total) {
        const int32_t m[1] = {id(e0)};
        nh += visit<1, GBM>(t, sh, m, s, cidx, w0, alloc);
    }
    return nh;
}

// Expands the frontier's entries [first, first + cnt), 0 < cnt <= 4 * U, of a
// graph with row slots: eight lanes take a vertex: lane j reads word j of its
// 32-byte slot, four vertices to a load and U loads in flight, so a level of
// few vertices is one short chain of dependent steps: ring, slot, bitmap,
// atomic, ring.  (One lane a vertex, six ids a lane, took 3,500 cycles for a
// level of a few vertices on the 80^3 matrix.)  Rows longer than a slot are
// left to the caller: lane i gets the bounds (b, d) of vertex i, or d = 0.
template <int U, bool CG, bool GBM, class Alloc>
__device__ __forceinline__ int expand_slots(const Trav<GBM> &t, const SharedState &sh, int first, int cnt, bool in_ring, int wstart, int32_t s,
                                            int cidx, int w0, Tally &acc, Alloc alloc, int32_t &b, int32_t &d)
{
    const int lane = threadIdx.x & 31;
    const int j = lane & 7;
    const int32_t *const word = reinterpret_cast<const int32_t *>(sh.home.g.slot) + j;
    int32_t v[U], m[U];
#pragma unroll
    for (int u = 0; u < U; u++) {   // past the last vertex: the empty slot behind the others
        const int p = first + 4 * u + (lane >> 3);
        v[u] = sh.home.n;
        if (in_ring) v[u] = ring_get(t.f, p, first + cnt, sh.home.n);
        else if (p < first + cnt) v[u] = fr_get(t.f, sh.home.spill, p, wstart);
    }
#pragma unroll
    for (int u = 0; u < U; u++) m[u] = ld<CG>(word + 8 * (int64_t)v[u]);
    int32_t most = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {   // lane j = 0 sums degrees, j = 1 input degrees
        acc.slot += (uint32_t)m[u];
        most = max(most, m[u]);
    }
    b = d = 0;
    if (__any_sync(0xffffffffu, j == 0 && most > SLOT_NB)) {   // long rows are read from adj
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int own = __shfl_sync(0xffffffffu, m[u], lane & 24);
            const int deg = __shfl_sync(0xffffffffu, m[u], (lane & 3) << 3);
            const int off = __shfl_sync(0xffffffffu, m[u], ((lane & 3) << 3) + 1);
            if ((lane >> 2) == u && deg > SLOT_NB) { d = deg; b = off; }
            if (own > SLOT_NB) {
                if (j == 1) acc.slot += (uint32_t)(ld<CG>(sh.home.rawdeg + v[u]) - m[u]);
                m[u] = -1;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++)
        if (j < 2) m[u] = -1;
    return visit<U, GBM>(t, sh, m, s, cidx, w0, alloc);
}

// Expands 32 vertices of a large level of a graph with row slots: a lane a
// vertex, six ids a lane -- fewer instructions a vertex, where every warp is
// busy.  v: the lane's vertex, or n, whose slot is empty.  next: its vertex of
// the warp's next 32; that slot comes into L1 beside this step's bitmap
// accesses.  A step is a chain of memory round trips (frontier, slot, bitmap
// and, for long rows, ids and bitmap again) which only the warps of one
// traversal share: with the frontier and the slot of the next step under way, no
// ring arithmetic past the ring, and a search instead of a loop for the long
// rows, the traversal of all of an 864,008-line bordered matrix takes 14.2 ms
// and not 17.4 (80^3 counts 3.95 and 4.09).
template <bool CG, bool GBM, class Alloc>
__device__ __forceinline__ int expand_wide(const Trav<GBM> &t, const SharedState &sh, int32_t v, int32_t next, int32_t s, int cidx,
                                           int w0, Tally &acc, Alloc alloc)
{
    const int4 sl0 = ld4<CG>(sh.home.g.slot + 2 * (int64_t)v), sl1 = ld4<CG>(sh.home.g.slot + 2 * (int64_t)v + 1);
    int32_t b = sl0.y, d = sl0.x;
    int32_t m[SLOT_NB] = {-1, -1, -1, -1, -1, -1};
    acc.edges += (unsigned)d;
    if (d <= SLOT_NB) {   // ids past the degree are -1 in the slot
        acc.einsp += (unsigned)b;
        m[0] = sl0.z; m[1] = sl0.w; m[2] = sl1.x; m[3] = sl1.y; m[4] = sl1.z; m[5] = sl1.w;
        d = 0;
    } else if (sh.home.pass == 0) {
        acc.einsp += (unsigned)ld<CG>(sh.home.rawdeg + v);
    }
    if (!CG) asm volatile("prefetch.global.L1 [%0];" ::"l"(sh.home.g.slot + 2 * (int64_t)next));
    int nh = visit<SLOT_NB, GBM>(t, sh, m, s, cidx, w0, alloc);
    if (__any_sync(0xffffffffu, d != 0)) nh += expand_edges<CG, GBM>(t, sh, b, d, s, cidx, w0, alloc);
    return nh;
}

// Expands the frontier's entries [first, first + cnt), 0 < cnt <= 32 (with row
// slots, 16), which were written while the level starting at wstart ran.
template <bool CG, bool GBM, class Alloc>
__device__ __forceinline__ int expand(const Trav<GBM> &t, const SharedState &sh, int first, int cnt, int wstart, int32_t s, int cidx, int w0,
                                      Tally &acc, Alloc alloc)
{
    const int lane = threadIdx.x & 31;
    const bool in_ring = first + cnt - wstart <= t.f.ring_size;
    int32_t b = 0, d = 0;
    int nh = 0;
    if (lane == 0) acc.xcnt += cnt;
    if (sh.home.g.slot != nullptr) {
        if (cnt <= 4) {
            nh = expand_slots<1, CG, GBM>(t, sh, first, cnt, in_ring, wstart, s, cidx, w0, acc, alloc, b, d);
        } else if (cnt <= 8) {
            nh = expand_slots<2, CG, GBM>(t, sh, first, cnt, in_ring, wstart, s, cidx, w0, acc, alloc, b, d);
        } else {
            nh = expand_slots<4, CG, GBM>(t, sh, first, cnt, in_ring, wstart, s, cidx, w0, acc, alloc, b, d);
        }
        if (!__any_sync(0xffffffffu, d != 0)) return nh;
    } else if (lane < cnt) {
        const int32_t v = fr_get(t.f, sh.home.spill, first + lane, wstart);
        b = ld<CG>(sh.home.g.ptr + v);
        d = ld<CG>(sh.home.g.ptr + v + 1) - b;
        acc.edges += (unsigned)d;
        if (sh.home.pass == 0) acc.einsp += (unsigned)ld<CG>(sh.home.rawdeg + v);
    }
    return nh + expand_edges<CG, GBM>(t, sh, b, d, s, cidx, w0, alloc);
}

// The helper warps: levels from [start, end) on (entries written while the
// level starting at wstart ran) until one is small enough for the leader
// alone.  One barrier a level.  The level counters rotate through three phases
// that run on from call to call (every warp counts them in `phase`): a level
// counts the next one's entries in tailc[phase] and its own dynamic fetches in
// fetch[phase]; the counters of the phase after next are cleared behind the
// level's barrier, when every warp is done with them.
template <int GT, bool CG, bool GBM>
__device__ __forceinline__ void run_levels(const Trav<GBM> &t, SharedState &sh, int htid, int bar, int &phase,
                                           Tally &acc)
{
    constexpr int NW = GT / 32 - 1;
    const int lane = htid & 31, wid = htid >> 5;
    const int32_t s = sh.src;
    const int cidx = sh.cidx;
    int start = sh.lv_start, end = sh.lv_end, wstart = sh.lv_wstart;
    int nlev = 0;
    for (;;) {
        int *const tailp = &sh.tailc[phase], *const fetchp = &sh.fetch[phase];
        const int cnt = end - start;
        // vertices a warp takes at a time: fewer than its lanes could, while
        // that keeps every warp busy
        const int take = sh.home.g.slot == nullptr ? min(32, max(1, (cnt + NW - 1) / NW))
                         : cnt <= 4 * NW     ? 4
                         : cnt <= 8 * NW     ? 8
                         : cnt <= 32 * NW    ? 16
                                             : 32;
        auto alloc = [&](int k) {
            int p = 0;
            if (lane == 0) p = atomicAdd(tailp, k);
            return end + __shfl_sync(0xffffffffu, p, 0);
        };
        int nh = 0;
        int base = wid * take;   // the first one by position, the others by demand
        auto more = [&]() {
            int p = 0;
            if (lane == 0) p = atomicAdd(fetchp, take);
            return __shfl_sync(0xffffffffu, p, 0) + NW * take;
        };
        if (sh.home.g.slot != nullptr && take == 32) {   // cnt > 32 * NW
            auto vertex = [&](int at) {
                return at + lane < cnt ? fr_get(t.f, sh.home.spill, start + at + lane, wstart) : sh.home.n;
            };
            int32_t v = vertex(base);
            while (base < cnt) {
                if (lane == 0) acc.xcnt += min(32, cnt - base);
                base = more();
                const int32_t next = vertex(base);
                nh += expand_wide<CG, GBM>(t, sh, v, next, s, cidx, start, acc, alloc);
                v = next;
            }
        } else {
            while (base < cnt) {
                nh += expand<CG, GBM>(t, sh, start + base, min(take, cnt - base), wstart, s, cidx, start, acc, alloc);
                if (cnt <= NW * take) break;
                base = more();
            }
        }
        if (lane == 0 && nh) atomicAdd(&sh.nh, nh);
        helper_sync<GT>(bar);
        const int nn = sh.tailc[phase];
        nlev++;
        wstart = start;
        start = end;
        end += nn;
        const int next = phase == 2 ? 0 : phase + 1;
        if (htid == 0) {
            const int clr = next == 2 ? 0 : next + 1;
            sh.tailc[clr] = 0;
            sh.fetch[clr] = 0;
        }
        phase = next;
        if (nn <= SOLO_MAX) break;
    }
    if (htid == 0) {   // for the leader's own lanes
        sh.lv_start = start;
        sh.lv_end = end;
        sh.lv_wstart = wstart;
        sh.prof[0] += (unsigned long long)nlev;
    }
}

// Warps wid, wid + nw, ... clear the nonzero chunks of a traversal's bitmap and
// their summaries.  The summaries say where the set bits are, so a state that
// touches a few stretches of a large matrix costs those stretches only; 32
// second-level words are read at once.
template <bool GBM>
__device__ __forceinline__ void clear_state(const Bits<GBM> &b, int wid, int nw, int lane)
{
    const int s2 = summ2_words(b);
    for (int i0 = 0; i0 < s2; i0 += 32) {
        const uint32_t mine = i0 + lane < s2 ? b.get(summ2(b) + i0 + lane) : 0u;
        unsigned any = __ballot_sync(0xffffffffu, mine != 0u);
        for (int k = 0; any; any &= any - 1u, k++) {
            const int j = __ffs(any) - 1;
            uint32_t m = __shfl_sync(0xffffffffu, mine, j);
            if (k % nw != wid) continue;
            const int i = i0 + j;
            for (; m; m &= m - 1u) b.put((((i << 5) + __ffs(m) - 1) << 5) + lane, 0u);
            if ((i << 5) + lane < (b.words >> 5)) b.put(summ1(b) + (i << 5) + lane, 0u);
        }
    }
}

// The second level, once every warp has read it.
template <bool GBM>
__device__ __forceinline__ void clear_summ2(const Bits<GBM> &b, int lane)
{
    for (int i = lane; i < summ2_words(b); i += 32) b.put(summ2(b) + i, 0u);
}

// The helper warps copy bitmap words [lo, hi) into a snapshot.
template <int GT, bool GBM>
__device__ __forceinline__ void save_state(const Bits<GBM> &b, uint32_t *snap, int lo, int hi, int htid)
{
    uint4 *dst = reinterpret_cast<uint4 *>(snap);
    for (int i = (lo >> 2) + htid; i < (hi >> 2); i += GT - 32) dst[i] = b.get4(i);
}

// The helper warps add the snapshot of source st (words [lo, hi)) to
// the bitmap of source s, st < s: the new vertices between the two join the
// first level (they were above st, so nothing was expanded from them), those
// above s are counted in sh.nh.
template <int GT, bool GBM>
__device__ __forceinline__ void merge_state(const Trav<GBM> &t, const uint32_t *snap, int lo, int hi, int st, int s, int cidx,
                                            SharedState &sh, int htid)
{
    const int lane = htid & 31;
    const uint4 *src = reinterpret_cast<const uint4 *>(snap);
    const int ws = s >> 5;
    const uint32_t above_s = ~1u << (s & 31);   // in word ws
    int cnt = 0;
    const int hi4 = hi >> 2;
    for (int i0 = lo >> 2; i0 < hi4; i0 += GT - 32) {   // warp-uniform trips
        const int i = i0 + htid;
        uint4 v = make_uint4(0u, 0u, 0u, 0u), c = v;
        if (i < hi4) {
            v = __ldcg(src + i);
            c = t.bits.get4(i);
        }
        const uint32_t nb[4] = {v.x & ~c.x, v.y & ~c.y, v.z & ~c.z, v.w & ~c.w};
        const uint32_t old[4] = {c.x, c.y, c.z, c.w};
        if (nb[0] | nb[1] | nb[2] | nb[3]) {
            t.bits.put4(i, make_uint4(c.x | v.x, c.y | v.y, c.z | v.z, c.w | v.w));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int w = 4 * i + q;
                if (nb[q] == 0u) continue;
                mark_word(t.bits, w, old[q] == 0u);
                cnt += w > ws ? __popc(nb[q]) : (w == ws ? __popc(nb[q] & above_s) : 0);
                if (w <= ws && w >= (st >> 5)) {   // the few words between the two sources
                    uint32_t x = nb[q];
                    if (w == ws) x &= (1u << (s & 31)) - 1u;
                    if (w == (st >> 5)) x &= ~1u << (st & 31);
                    for (; x; x &= x - 1u) fr_put(t.f, sh.home.spill, atomicAdd(&sh.npush, 1), 0, (w << 5) + __ffs(x) - 1, true);
                }
            }
        }
        if (t.stamp != nullptr) {   // a word at a time across the warp (lane = bit)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                unsigned any = __ballot_sync(0xffffffffu, nb[q] != 0u);
                for (; any; any &= any - 1u) {
                    const int j = __ffs(any) - 1;
                    const uint32_t x = __shfl_sync(0xffffffffu, nb[q], j);
                    const int32_t m = ((4 * (i - lane + j) + q) << 5) + lane;
                    if (((x >> lane) & 1u) && m > s - cidx) t.stamp[m] = (uint16_t)cidx;
                }
            }
        }
    }
    cnt = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
    if (lane == 0 && cnt) atomicAdd(&sh.nh, cnt);
}

// Writes lists first .. len - 1 of a chain -- sources s0, s0 + 1, .. which share
// one bitmap -- by the helper warps, while the leader goes on with the next
// sources: it waits only until the set vertices are out of the bitmap (the
// barrier in the middle), unless the traversal has no scratch for both
// (JobArgs::stamp_other).  Bits are only ever added along a chain, so list i is
// { v > s0 + i : v set, stamp(v) <= i } once source i is done; what later
// sources add has larger stamps.  One exact pool
// range holds all of the chain's lists (one global atomic per chain).
//
// First each warp extracts its share of the bitmap's chunks, in order, into
// `lists` (offsets from a count pass).  Then the lists go out 32 at a time:
// every warp takes a block of the extracted vertices; a vertex belongs to the
// lists [stamp, v - s0) of the chain, so two counters a vertex, summed, give
// each warp its block's entries in each list and, over the warps, where they
// start; then the block's vertices are read once more and, 32 at a time, go to
// each of the lists by ballot -- where all 32 belong to all of the lists, as
// most do, as one full store a list.  (A warp a list, filtering the last list
// once per list with a dependent load of the stamp in every step, took 1,650
// cycles a source on the 80^3 matrix with all warps waiting for it.)
// Lists of pass G^T (columns of L) also count their entries into the L row
// histogram, one reduction for the 32 lists.
template <int GT, bool GBM>
__device__ __forceinline__ void write_lists(const JobArgs &a, const Trav<GBM> &t, SharedState &sh, int (*hist)[32],
                            int htid, int bar)
{
    constexpr int NH = GT / 32 - 1;
    constexpr int UNR = 4;
    const int lane = htid & 31, wid = htid >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int s0 = sh.chain_s0, first = sh.chain_first, len = sh.chain_len, chain_hi = sh.chain_hi;
    const int64_t total = sh.chain_total;
    const uint16_t *const stamp = sh.stamp;
    int32_t *const scratch = sh.home.lists;
    const int64_t row0 = sh.home.row + s0;   // cnt / poff entry of s0
    int32_t *const lrow = sh.home.lrow;

    // past the pool's capacity the chain's lists are not written, the tail
    // still advances, and its final value is the capacity the job needs
    long long base = 0;
    if (wid == 0 && lane == 0 && total > 0) {
        const unsigned long long o = atomicAdd(a.pool_tail, (unsigned long long)total);
        base = (int64_t)o + total <= a.pool_cap ? (long long)o : -1;
        if (base < 0) atomicOr(a.status, ERR_POOL_OVERFLOW);
    }

    // set bits above the first list's source: words from w0 on (first_mask on w0)
    const int w0 = (s0 + first + 1) >> 5;
    const uint32_t first_mask = ~0u << ((s0 + first + 1) & 31);
    const int c_lo = w0 >> 5;
    const int c_hi = chain_hi > s0 + first ? (chain_hi >> 10) + 1 : c_lo;
    const int share = (max(c_hi - c_lo, 0) + NH - 1) / NH;
    const int my_lo = c_lo + wid * share, my_hi = min(c_hi, my_lo + share);
    auto word = [&](int cc) {
        const int w = (cc << 5) + lane;
        uint32_t x = t.bits.get(w);
        if (w < w0) x = 0u;
        if (w == w0) x &= first_mask;
        return x;
    };
    int mine = 0;
    if (my_lo < my_hi)
        for_nonzero_chunks<GBM>(t.bits, my_lo, my_hi, [&](int cc) { mine += __popc(word(cc)); });
    mine = (int)__reduce_add_sync(0xffffffffu, (unsigned)mine);
    if (lane == 0) sh.warp[wid] = mine;
    helper_sync<GT>(bar);
    int pos = 0, all = 0;
    for (int k = 0; k < NH; k++) {
        const int c = (int)sh.warp[k];
        pos += k < wid ? c : 0;
        all += c;
    }
    if (my_lo < my_hi)
        for_nonzero_chunks<GBM>(t.bits, my_lo, my_hi, [&](int cc) {
            uint32_t x = word(cc);
            const int pc = __popc(x);
            int incl = pc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int excl = incl - pc;
            // at most two entries a word: a word per lane; denser chunks a
            // word at a time across the warp (lane = bit)
            if (__reduce_max_sync(0xffffffffu, (unsigned)pc) <= 2u) {
                for (int at = pos + excl; x; x &= x - 1u, at++) scratch[at] = (((cc << 5) + lane) << 5) + __ffs(x) - 1;
            } else {
                for (unsigned nzw = __ballot_sync(0xffffffffu, x != 0u); nzw; nzw &= nzw - 1u) {
                    const int j = __ffs(nzw) - 1;
                    const uint32_t xj = __shfl_sync(0xffffffffu, x, j);
                    const int pj = __shfl_sync(0xffffffffu, excl, j);
                    if ((xj >> lane) & 1u) scratch[pos + pj + __popc(xj & below)] = (((cc << 5) + j) << 5) + lane;
                }
            }
            pos += __shfl_sync(0xffffffffu, incl, 31);
        });
    if (wid == 0 && lane == 0) sh.pool_base = base;
    gsync<GT>(bar);   // the bitmap is free, the vertices are out
    base = sh.pool_base;

    const int steps = (all + 31) >> 5, per = (steps + NH - 1) / NH;
    const int k_lo = min(all, wid * per * 32), k_hi = min(all, k_lo + per * 32);
    long long carry = 0;
    for (int i0 = first; i0 < len; i0 += 32) {
        const int nl = min(32, len - i0);
        // lane l: list i0 + l, its entries and its place
        const int c = lane < nl ? a.cnt[row0 + i0 + lane] : 0;
        long long incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        long long p = base + carry + incl - c;
        carry += __shfl_sync(0xffffffffu, incl, 31);
        if (wid == 0 && lane < nl) a.poff[row0 + i0 + lane] = base >= 0 ? p : -1;
        if (base < 0) continue;
        // the lists [lo, hi) of the 32 that vertex v belongs to
        auto lists_of = [&](int32_t v, int st, int &lo, int &hi) {
            lo = max(st - i0, 0);
            hi = v - s0 - i0;
        };
        hist[wid][lane] = 0;
        __syncwarp();
        int whole = 0;   // vertices that belong to all 32
        for (int k0 = k_lo; k0 < k_hi; k0 += 32 * UNR) {
            int32_t v[UNR];
            int st[UNR];
#pragma unroll
            for (int u = 0; u < UNR; u++) v[u] = k0 + 32 * u + lane < k_hi ? __ldcg(scratch + k0 + 32 * u + lane) : -1;
#pragma unroll
            for (int u = 0; u < UNR; u++) st[u] = v[u] > s0 && v[u] <= chain_hi ? (int)stamp[v[u]] : INT32_MAX;
#pragma unroll
            for (int u = 0; u < UNR; u++) {
                int lo, hi;
                lists_of(v[u], min(st[u], 1 << 20), lo, hi);
                const bool full = lo == 0 && hi >= 32;
                whole += __popc(__ballot_sync(0xffffffffu, full));
                if (!full && lo < 32 && hi > lo) {
                    atomicAdd(&hist[wid][lo], 1);
                    if (hi < 32) atomicAdd(&hist[wid][hi], -1);
                }
            }
        }
        __syncwarp();
        int n = hist[wid][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, n, o);
            if (lane >= o) n += y;
        }
        n += whole;
        __syncwarp();
        hist[wid][lane] = n;
        helper_sync<GT>(bar);
        int sum = 0;
        for (int k = 0; k < NH; k++) {
            const int x = hist[k][lane];
            p += k < wid ? x : 0;
            sum += x;
        }
        // a list's running count and its vertices disagree: an internal fault,
        // and nothing is written
        const bool bad = __any_sync(0xffffffffu, lane < nl && sum != c);
        if (bad && lane == 0) atomicOr(a.status, ERR_COUNT_MISMATCH);
        for (int k0 = bad ? k_hi : k_lo; k0 < k_hi; k0 += 32 * UNR) {
            int32_t v[UNR];
            int st[UNR];
#pragma unroll
            for (int u = 0; u < UNR; u++) v[u] = k0 + 32 * u + lane < k_hi ? __ldcg(scratch + k0 + 32 * u + lane) : -1;
#pragma unroll
            for (int u = 0; u < UNR; u++) st[u] = v[u] > s0 && v[u] <= chain_hi ? (int)stamp[v[u]] : INT32_MAX;
#pragma unroll
            for (int u = 0; u < UNR; u++) {
                int lo, hi;
                lists_of(v[u], min(st[u], 1 << 20), lo, hi);
                if (lrow && lo < nl) {
                    const int k = min(hi, nl) - lo;
                    if (k > 0) atomicAdd(lrow + v[u], k);
                }
                if (__all_sync(0xffffffffu, lo == 0 && hi >= nl)) {
#pragma unroll 4
                    for (int l = 0; l < nl; l++) a.pool[__shfl_sync(0xffffffffu, p, l) + lane] = v[u];
                    p += 32;
                } else {
                    int got = 0;
                    for (int l = 0; l < nl; l++) {
                        const bool in = lo <= l && l < hi;
                        const unsigned bal = __ballot_sync(0xffffffffu, in);
                        const long long q = __shfl_sync(0xffffffffu, p, l);
                        if (in) a.pool[q + __popc(bal & below)] = v[u];
                        if (lane == l) got = __popc(bal);
                    }
                    p += got;
                }
            }
        }
        helper_sync<GT>(bar);   // the counters are free again
    }
    // Streaming: count the chain's entries into the pool blocks they fill.
    // Every list of the chain is written (the barrier above); one fence makes
    // those writes visible device-wide before the counts that let the host
    // copy a full block out while the traversals go on.
    if (a.blk_done != nullptr && wid == 0 && lane == 0 && total > 0 && base >= 0) {
        __threadfence();
        const int64_t end = base + total;
        const int64_t bsz = (int64_t)1 << a.blk_shift;
        for (int64_t b = base >> a.blk_shift; b <= (end - 1) >> a.blk_shift; b++) {
            const int64_t lo = max(base, (long long)(b * bsz)), hi = min(end, (b + 1) * bsz);
            atomicAdd(a.blk_done + b, (unsigned int)(hi - lo));
        }
    }
}

// One op of the leader's, run by the helper warps (htid: the thread among
// them) behind the traversal's barrier; a second one tells the leader that it
// is done.
template <int GT, bool CG, bool GBM, bool LISTS>
__device__ __forceinline__ void run_op(const JobArgs &a, Trav<GBM> &t, SharedState &sh,
                                       int (*hist)[32], int op, int htid, int bar, int &phase, Tally &acc)
{
    if (LISTS) t.stamp = sh.stamp;
    if (op == OP_LEVELS) {
        carry(sh, acc, htid & 31);
        __syncwarp();
        run_levels<GT, CG, GBM>(t, sh, htid, bar, phase, acc);
    } else if (op == OP_CLEAR) {
        clear_state<GBM>(t.bits, htid >> 5, GT / 32 - 1, htid & 31);
    } else if (op == OP_SAVE) {
        save_state<GT, GBM>(t.bits, sh.home.snaps + (int64_t)sh.snap * a.bitmap_words, sh.lo, sh.hi, htid);
    } else if (op == OP_MERGE) {
        merge_state<GT, GBM>(t, sh.home.snaps + (int64_t)sh.snap * a.bitmap_words, sh.lo, sh.hi, sh.t, sh.src, sh.cidx, sh,
                             htid);
    } else if (LISTS && op == OP_LISTS) {
        write_lists<GT, GBM>(a, t, sh, hist, htid, bar);   // the leader goes on from its middle
        if (a.stamp_other != 0) return;
    }
    gsync<GT>(bar);
}

// Nonzero stretch of a bitmap as words [lo, hi), whole chunks, and its number
// of nonzero chunks; one warp.
template <bool GBM>
__device__ __forceinline__ int state_extent(const Bits<GBM> &b, int lane, int &lo, int &hi)
{
    int first = INT32_MAX, last = -1, chunks = 0;
    for (int i = lane; i < summ2_words(b); i += 32) {
        const uint32_t m = b.get(summ2(b) + i);
        if (m) {
            first = min(first, (i << 5) + __ffs(m) - 1);
            last = (i << 5) + 31 - __clz(m);
            chunks += __popc(m);
        }
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    lo = last < 0 ? 0 : first << 5;
    hi = (last + 1) << 5;
    return (int)__reduce_add_sync(0xffffffffu, (unsigned)chunks);
}

// The CTA's next sources, from s on: those of the units that `claim` claimed
// (lane 0 of the first leader).  Returns where they end: s when there are none.
template <class C>
__device__ __noinline__ int32_t next_units(int32_t s, int half)
{
    if (half == 0 && (threadIdx.x & 31) == 0) {
        SharedState &sh = cta<C>().t[0];
        const SharedPiece &own = sh.own;
        const unsigned long long claim = sh.claim;
        const int unit = (int)(claim & UNIT_MASK), end = (int)((claim >> UNIT_BITS) & UNIT_MASK);
        if (unit < end) {
            const int take = sh.claimed, next = min(unit + take, end);
            sh.next_end = min(own.first + next * UNIT, own.last);
            const int more = min(max((end - next) >> 3, 1), CLAIM_MAX);
            sh.claimed = more;
            const unsigned now = clock32() >> 8;   // in 256 cycles, 24 bits
            const int done = s - own.s_lo;         // sources since the piece began
            if (done > 0) {
                const unsigned took = (now - sh.unit_t) & 0xffffffu;
                if (sh.unit_done == 0) {   // the first unit
                    sh.unit_most = took;
                    own.fresh[0] = max(took, 1u);
                    sh.unit_sum = 0u;
                    sh.unit_mean = took;
                } else {
                    const int units = (done - sh.unit_done + UNIT - 1) / UNIT;
                    const unsigned usual = (unsigned)units * sh.unit_mean;
                    // a traversal from nothing in the middle of a piece of small ones is
                    // not what the next units will take; up to sixteenfold they vary (a
                    // limit of four hid what was left of the power-law matrices' pieces:
                    // 200K lines 19.3 ms, now 17.1)
                    const bool spike = took > 16 * usual;
                    if (spike) sh.unit_most = max(sh.unit_most, took - usual);
                    sh.unit_sum += spike ? usual : took;
                    sh.unit_mean = max((unsigned)__fdividef((float)sh.unit_sum * (float)UNIT, (float)(done - UNIT)), 1u);
                    *reinterpret_cast<volatile unsigned long long *>(own.cost) =
                        (unsigned long long)sh.unit_most << 32 | sh.unit_mean;
                }
                sh.unit_done = done;
            }
            sh.unit_t = now;
            // last: the store waits for the claim, which is needed a claim later
            sh.claim = atomicAdd(own.word, (unsigned long long)more);
        } else {
            sh.next_end = s;
        }
    }
    pair_sync();
    return cta<C>().t[0].next_end;
}

// Where the cost of a piece that begins at `line` is noted.
constexpr int FRESH_BUCKETS = 1024;

__device__ __forceinline__ int fresh_bucket(int64_t line, int64_t lines)
{
    return (int)min(line * FRESH_BUCKETS / max(lines, (int64_t)1), (int64_t)FRESH_BUCKETS - 1);
}

// A part of another CTA's piece, as a piece word, or 0: of the parts of x units
// from the top, half of what is left less half of what starting afresh costs,
// the one that saves most.  While there is none but some CTA has yet to show
// what its units cost, it looks again (a bounded number of times; every CTA of
// the launch is resident and goes on).  One warp.
template <class C>
__device__ __noinline__ unsigned long long take_part(int ctas, int lane)
{
    const JobArgs &a = cta<C>().a;
    for (int attempt = 0; attempt < (1 << 22); attempt++) {
        bool wait = false;
        unsigned best = 0u;
        int from = -1, best_x = 0;
        unsigned long long best_w = 0ull;
        for (int c = lane; c < ctas; c += 32) {
            const unsigned long long w = __ldcg(a.shared_piece + c), cost = __ldcg(a.shared_cost + c);
            const long long left = (long long)((w >> UNIT_BITS) & UNIT_MASK) - (long long)(w & UNIT_MASK);
            const long long mean = (long long)(cost & 0xffffffffull);
            long long extra = (long long)(cost >> 32);
            if (left <= 0) continue;
            if (mean == 0) { wait = true; continue; }
            if (left * mean <= extra) continue;
            {   // a traversal from nothing above the middle: as the next piece there found it
                const Range &rg = a.ranges[w >> (2 * UNIT_BITS)];
                const int64_t line0 = a.mats[rg.mat].line_base + rg.offset;
                const int64_t mid = line0 + ((int64_t)((w >> UNIT_BITS) & UNIT_MASK) - left / 2) * UNIT;
                int b = fresh_bucket(mid, a.L);
                const int b_end = min(fresh_bucket(line0 + rg.nj, a.L), b + 64);
                unsigned f = 0u;
                for (; b <= b_end && f == 0u; b++) f = __ldcg(a.fresh_cost + b);
                extra = max(extra, (long long)f);
            }
            const long long x = (left * mean - extra) / (2 * mean);
            if (x < 1) continue;
            const unsigned gain = (unsigned)min(x * mean, 0x7fffffffll);
            if (gain > best) { best = gain; from = c; best_x = (int)x; best_w = w; }
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best);
        if (top == 0u) {
            if (!__any_sync(0xffffffffu, wait)) return 0ull;
            __nanosleep(1000);
            continue;
        }
        const int who = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
        unsigned long long got = 0ull;
        if (lane == who) {
            const int end = (int)((best_w >> UNIT_BITS) & UNIT_MASK), range = (int)(best_w >> (2 * UNIT_BITS));
            const unsigned long long rest = piece_word(range, end - best_x, (int)(best_w & UNIT_MASK));
            if (atomicCAS(a.shared_piece + from, best_w, rest) == best_w) got = piece_word(range, end, end - best_x);
        }
        got = __shfl_sync(0xffffffffu, got, who);
        if (got) return got;   // else the owner, or another CTA, was there first
    }
    return 0ull;
}

// The sources s_lo, s_lo + stride, ... < s_hi of one work piece, in order,
// each starting from the previous source's state whenever that is valid.
//
// A traversal's first warp, its leader, runs the sources by itself: nine of
// ten on nested-dissection matrices add no vertex below the source and need no
// other warp.  The other warps wait at the traversal's barrier and join only
// for large steps: a level of more than SOLO_MAX vertices (and the levels after
// it while they stay large), clearing or copying a wide bitmap, a chain's list
// output.  With all warps at a barrier two or three times a source, the 80^3
// counts spent 4,600 cycles a source and pass.
//
// PAIRED: the leaders of the two passes exchange "s+1 reached" flags after
// every source (pair_sync).  s-1 is in X_G(s) exactly when s is in
// hi_{G^T}(s-1), and then X(s-1) u {s-1} is inside X(s) and hi(s-1) minus {s}
// inside hi(s), so the bitmap can be kept.  The same holds for every earlier
// source t: when s is in hi_{G^T}(t), the state that pass G had after t is
// inside that of s.  States that took a long traversal to build are copied to
// global memory (snapshots, the SNAP_MAX latest of a piece) with the other
// pass's bits for the sources after t, and each later source takes over the
// snapshots that it provably contains.  On power-law matrices nearly half of
// the sources do not contain s-1 but do contain some t a few lines below, whose
// closure is most of the matrix: the 20,000-line one inspects 2.4e7 edges
// instead of 2.7e8.
template <int BLOCK, bool PAIRED, bool CG, bool GBM, bool LISTS = true>
__device__ __noinline__ void lead_piece(Trav<GBM> t, int32_t s_lo, int32_t s_hi, int32_t stride, bool shared, int half)
{
    using C = CtaOf<BLOCK, PAIRED, LISTS>;
    constexpr int GT = PAIRED ? BLOCK / 2 : BLOCK;
    static_assert(GT >= 64, "a leader and at least one helper");
    const JobArgs &a = cta<C>().a;
    SharedState *const shs = cta<C>().t;
    volatile int (*const pair_flag)[2] = cta<C>().pair_flag;
    const int bar = 1 + half;
    SharedState &sh = shs[half];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int pass = sh.home.pass;
    const int32_t n = sh.home.n;
    Tally acc;
    const int nsnap = PAIRED ? a.snap_k : 0;
    auto collective = [&](int op) {   // arguments are in place
        if (lane == 0) {
            sh.op = op;
            if (LISTS) sh.stamp = t.stamp;
        }
        __syncwarp();
        gsync<GT>(bar);   // the helpers have the op
        gsync<GT>(bar);   // they are done
    };
    auto take_nh = [&]() {   // what the last op counted
        const int v = sh.nh;
        __syncwarp();
        if (lane == 0) sh.nh = 0;
        return v;
    };
    // tallies: the first lane's, in shared memory
    auto tally = [&](unsigned long long &x, unsigned long long v) { if (lane == 0) x += v; };
    auto spent = [&](int q, long long c0) {   // cycles of one kind, none of the sources' own
        const unsigned long long c = (unsigned long long)(clock64() - c0);
        tally(sh.prof[q], c);
        tally(sh.prof[1], 0ull - c);
    };
    tally(sh.prof[1], 0ull - (unsigned long long)clock64());
    uint32_t n_levels = 0;                // 2^32 levels would be a piece of half an hour
    uint32_t c_levels = 0, c_wait = 0;    // cycles in 256s

    int prev = -2;
    int cidx = -1;            // index of the last source in its chain (-1: none yet)
    int hc = 0;               // set bits above the last source
    unsigned xch = 0;         // exchanges with the other pass so far
    bool mine = false, other = false;   // this pass, the other pass reached s
    bool step = false;        // s is not for a run
    long long total = 0;      // entries of the chain's lists from `pending` on (up to 94 lists of n)
    int pending = 0;          // the chain's first list that is not written
    // the seeding window: lane i holds row bounds and degree of source wlo + i
    int wlo = 0, whi = 0, wb = 0, we = 0, wraw = 0, wadj0 = 0;
    if (lane < SNAP_MAX) sh.snap_t[lane] = -1;
    // A state of this many vertices is worth a copy of the bitmap (an eighth of
    // its words), and a copy is paid with as many vertices traversed or taken
    // over: where snapshots help, long traversals pay for them at once, and
    // where traversals are short they cost next to nothing.
    const int heavy = max(64, n >> 8);
    if (lane == 0) {
        sh.snaps = sh.weight = 0;
        if (sh.snap_credit < 0) sh.snap_credit = 4 * heavy;
    }
    __syncwarp();

    auto lists_out = [&]() {   // of the chain's sources since `pending`
        const long long c0 = clock64();
        int lo, hi;
        state_extent<GBM>(t.bits, lane, lo, hi);
        if (lane == 0) {
            sh.chain_s0 = prev - cidx;
            sh.chain_first = pending;
            sh.chain_len = cidx + 1;
            sh.chain_total = total;
            sh.chain_hi = min(hi << 5, n) - 1;
        }
        collective(OP_LISTS);
        if (a.stamp_other == 0) gsync<GT>(bar);   // its stamps and its queue are free again
        pending = cidx + 1;
        total = 0;
        spent(5, c0);
    };
    auto end_chain = [&]() {
        int lo, hi;
        if (LISTS && a.want_pattern) {
            if (pending <= cidx) lists_out();
            // the helpers read this chain's stamps on: the next chain takes
            // the traversal's other row
            t.stamp = t.stamp == sh.home.stamps ? sh.home.stamps + a.stamp_other : sh.home.stamps;
        }
        const long long c0 = clock64();
        const int chunks = state_extent<GBM>(t.bits, lane, lo, hi);
        if (chunks <= 48) {
            clear_state<GBM>(t.bits, 0, 1, lane);
            __syncwarp();
        } else {
            collective(OP_CLEAR);
        }
        clear_summ2(t.bits, lane);
        __syncwarp();
        if (GBM) __threadfence_block();
        spent(6, c0);
    };

    if (PAIRED && shared && half == 0 && lane == 0) {
        sh.claim = atomicAdd(sh.own.word, 1ull);   // a claim ahead of the sources
        sh.claimed = 1;
        sh.unit_t = clock32() >> 8;
        sh.unit_done = 0;
    }
    if (lane == 0) sh.own.s_lo = s_lo;
    for (int32_t s = s_lo;;) {
        if (PAIRED && s >= s_hi && shared) s_hi = next_units<C>(s, half);
        const bool more = s < s_hi;   // else: end the piece's last chain
        // a long chain's lists go out as it grows, not all at its end
        if (LISTS && a.want_pattern && cidx - pending >= 63 && total >= 1 << 15) lists_out();
        // a new seeding window when s is past the current one (consecutive
        // sources only): row bounds, then the rows themselves
        if (more && stride == 1 && s >= whi) {
            const int cnt = min(s_hi - s, SEED_WIN);
            const int i = min(lane, cnt - 1);
            wb = ld<CG>(sh.home.g.ptr + s + i);
            we = ld<CG>(sh.home.g.ptr + s + i + 1);
            if (pass == 0) wraw = ld<CG>(sh.home.rawdeg + s + i);
            wadj0 = __shfl_sync(0xffffffffu, wb, 0);
            const int k = __popc(__ballot_sync(0xffffffffu, lane < cnt && we - wadj0 <= SEED_ADJ));   // rows that fit
            const int na = k ? __shfl_sync(0xffffffffu, we, k - 1) - wadj0 : 0;
            __syncwarp();
            const int32_t *const from = sh.home.g.adj + wadj0;
#pragma unroll 1
            for (int q0 = lane; q0 < na; q0 += 256) {   // 256 ids in flight: one round trip for most windows
                int32_t x[8];
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] = q0 + 32 * u < na ? ld<CG>(from + q0 + 32 * u) : 0;
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (q0 + 32 * u < na) sh.win_adj[q0 + 32 * u] = x[u];
            }
            __syncwarp();
            wlo = s;
            whi = s + k;   // k == 0: a row too long for the window, read where it lies
        }
        const bool in_win = stride == 1 && s < whi;

        // A run: the sources from s on that both passes' chains reach and that
        // add no vertex below themselves, in one go.  New ids of the window's
        // rows from s on are collected in row order, at most 32 of them; the
        // first source to hold an id sets it.  The run ends before the first
        // source that some new id lies below (it needs a traversal), or that
        // either pass has not reached (its chain ends there): each pass says
        // which of the sources are set when their turn comes (run_set) and
        // where its run would end, and the shorter of the two is taken.
        // On the 80^3 matrix 85% of the sources go in runs of about seven, at
        // some 150 cycles a source instead of the 1,600 that the step below
        // takes (counts 8.9 ms to 5.2 ms).
        // Both passes come here or neither does; one that cannot run (a row too
        // long for its window, a chain near its last stamp) says k = 0.
        if (PAIRED && more && mine && other && !step) {
            const bool can = in_win && !(a.want_pattern && cidx + 32 >= 65535);
            int k = can ? min(whi - s, 31) : 0;
            const int i0 = can ? s - wlo : 0;
            const int p0 = __shfl_sync(0xffffffffu, wb, i0) - wadj0;
            const int p1 = can ? __shfl_sync(0xffffffffu, we, i0 + k - 1) - wadj0 : p0;
            const uint32_t ws = s + lane < n ? t.bits.get((s + lane) >> 5) : 0u;
            unsigned run_set = __ballot_sync(0xffffffffu, (ws >> ((s + lane) & 31)) & 1u);
            int ne = 0;
            for (int q0 = p0; q0 < p1 && ne <= 32; q0 += 128) {
                int32_t x[4];
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = q0 + 32 * u + lane < p1 ? sh.win_adj[q0 + 32 * u + lane] : -1;
#pragma unroll
                for (int u = 0; u < 4; u++) w[u] = x[u] >= 0 ? t.bits.get(x[u] >> 5) : ~0u;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const bool isnew = !((w[u] >> (x[u] & 31)) & 1u);
                    const unsigned bal = __ballot_sync(0xffffffffu, isnew);
                    const int at = ne + __popc(bal & below);
                    if (isnew && at <= 32) {
                        sh.ev_x[at] = x[u];
                        sh.ev_p[at] = q0 + 32 * u + lane;
                    }
                    ne += __popc(bal);
                }
            }
            __syncwarp();
            // the row (source s + ei) of event `lane`, and of the 33rd, where
            // the run must end: the last row that begins at or before it
            const int x = lane < ne ? sh.ev_x[lane] : -1;
            auto row_of = [&](int p) {
                int o = i0;   // rows begin in order
#pragma unroll
                for (int h = 16; h; h >>= 1) {
                    const int c = o + h;
                    const int v = __shfl_sync(0xffffffffu, wb, min(c, 31)) - wadj0;
                    if (c < i0 + k && v <= p) o = c;
                }
                return o - i0;
            };
            const int ei = row_of(lane < ne ? sh.ev_p[lane] : 0);
            int cut = k;
            if (ne > 32) cut = min(cut, row_of(sh.ev_p[32]));
            bool win = false;
            if (ne > 0) {
                const unsigned same = __match_any_sync(0xffffffffu, lane < ne ? x : -1 - lane);
                win = lane < ne && !(same & below);
                cut = min(cut, (int)__reduce_min_sync(0xffffffffu, win && x < s + ei ? (unsigned)ei : 32u));
                run_set |= __reduce_or_sync(0xffffffffu, win && x > s + ei && x - s < 32 ? 1u << (x - s) : 0u);
            }
            const int par = xch & 1;
            xch++;
            if (lane == 0) {
                pair_flag[par][half] = (int)run_set;
                sh.run_cut[par] = cut | k << 8;
            }
            pair_sync();
            const unsigned oset = (unsigned)pair_flag[par][1 - half];
            const int ocut = shs[1 - half].run_cut[par];
            cut = min(cut, ocut & 0xff);
            k = min(k, ocut >> 8);
            // sources s .. s + cut - 1: set in both passes, and none below
            const unsigned both = run_set & oset;
            if (~both) cut = min(cut, __ffs(~both) - 1);
            if (cut > 0) {
                win = win && ei < cut;
                uint32_t w = win ? 0u : ~0u;
                t.bits.add(t.bits.place(x), 1u << (x & 31), w);
                mark_word(t.bits, x >> 5, w == 0u);
                if (win && t.stamp != nullptr) t.stamp[x] = (uint16_t)(cidx + 1 + ei);
                // lane i: source s + i; events are in row order
                const unsigned wins = __ballot_sync(0xffffffffu, win);
                int upto = 0;   // events of rows 0 .. lane
                if (wins) {
                    const int key = lane < ne ? ei : 64;
#pragma unroll
                    for (int h = 16; h; h >>= 1)
                        if (__shfl_sync(0xffffffffu, key, upto + h - 1) <= lane) upto += h;
                    if (__shfl_sync(0xffffffffu, key, upto) <= lane) upto++;   // all 32
                }
                const int found = upto >= 32 ? __popc(wins) : __popc(wins & ((1u << upto) - 1u));
                const int c = hc + found - (lane + 1);
                const int deg = __shfl_sync(0xffffffffu, we - wb, (i0 + lane) & 31);
                const int raw = __shfl_sync(0xffffffffu, wraw, (i0 + lane) & 31);
                if (lane < cut) {
                    const int64_t slot = sh.home.row + s + lane;
                    a.cnt[slot] = c;
                    a.nxt[slot] = (uint8_t)((run_set >> (lane + 1)) & 1u);
                    acc.edges += (unsigned)deg;
                    if (pass == 0) acc.einsp += (unsigned)raw;
                }
                if (LISTS) total += (long long)cut * hc - cut * (cut + 1) / 2 +
                         (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < cut ? found : 0));
                hc = __shfl_sync(0xffffffffu, c, cut - 1);
                cidx += cut;
                prev = s + cut - 1;
                mine = (run_set >> cut) & 1u;
                other = (oset >> cut) & 1u;
                s += cut;
            }
            // where a window or its 31 sources ended, another run may follow;
            // else s is a source that ended the run
            step = cut == 0 || cut < k;
            __syncwarp();
            if (cut > 0) continue;
        }
        step = false;
        int32_t b0 = 0, d0 = 0;
        if (in_win) {
            b0 = __shfl_sync(0xffffffffu, wb, s - wlo);
            d0 = __shfl_sync(0xffffffffu, we, s - wlo) - b0;
        } else if (more) {
            b0 = ld<CG>(sh.home.g.ptr + s);
            d0 = ld<CG>(sh.home.g.ptr + s + 1) - b0;
        }

        // take over the previous source's state, or end its chain; chain
        // indices are 16-bit stamps: a chain ends after 65535 sources
        bool reuse = false;
        if (more && a.reuse && prev == s - 1 && !(a.want_pattern && cidx + 1 >= 65535)) {
            if (PAIRED) {
                reuse = other;
            } else {
                bool hit = false;
                for (int k = lane; k < d0; k += 32)
                    hit |= (in_win ? sh.win_adj[b0 - wadj0 + k] : ld<CG>(sh.home.g.adj + b0 + k)) == s - 1;
                reuse = __any_sync(0xffffffffu, hit);
            }
        }
        if (reuse) {
            cidx++;
        } else {
            if (cidx >= 0) end_chain();
            if (!more) {   // the next piece starts from an empty bitmap
                if (lane == 0) sh.nsrc += (unsigned)((s - sh.own.s_lo) / stride);
                break;
            }
            tally(sh.nfresh, 1u);
            cidx = 0;
            hc = 0;
            total = 0;
            pending = 0;
            if (nsnap > 0 && lane == 0) sh.weight = 0;
        }

        // Seeding: s itself (in the lane after its row) and its neighbours;
        // those below s are the first
        // level.  nh counts new vertices above s, and s when it is new: a
        // source that was set already was counted by the sources before it.
        int tail = 0, nh = 0;
        bool self = false;   // s is set
        auto alloc = [&](int k) { const int p = tail; tail += k; return p; };
        if (lane == 0) {
            acc.edges += (unsigned)d0;
            if (pass == 0 && !in_win) acc.einsp += (unsigned)ld<CG>(sh.home.rawdeg + s);
        }
        if (in_win && lane == s - wlo) acc.einsp += (unsigned)wraw;
        if (nsnap > 0 && sh.snaps > 0) {
            // the newest snapshot that s contains and its state does not yet,
            // until there is none (bit t set: t and all of its state are in)
            for (;;) {
                int st = -1;
                if (lane < nsnap) st = sh.snap_t[lane];
                if (st >= 0) {
                    const int w = (s >> 5) - (st >> 5);
                    if (!(w < SNAP_REACH && ((sh.snap_reach[lane][w] >> (s & 31)) & 1u) &&
                          !((t.bits.get(st >> 5) >> (st & 31)) & 1u)))
                        st = -1;
                }
                const int best = __reduce_max_sync(0xffffffffu, st);
                if (best < 0) break;
                const long long c0 = clock64();
                if (!self) {   // before the merge, which leaves it out
                    const int32_t m[1] = {lane == 0 ? s : -1};
                    nh += visit<1, GBM>(t, sh, m, s, cidx, 0, alloc);
                    self = true;
                }
                const int k = __ffs(__ballot_sync(0xffffffffu, st == best)) - 1;
                if (lane == 0) {
                    sh.weight = min(sh.weight + sh.snap_w[k], 1 << 28);
                    sh.snap_credit = min(sh.snap_credit + sh.snap_w[k], 1 << 28);
                    sh.src = s;
                    sh.cidx = cidx;
                    sh.snap = k;
                    sh.t = best;
                    sh.lo = sh.snap_lo[k];
                    sh.hi = sh.snap_hi[k];
                    sh.npush = tail;
                }
                collective(OP_MERGE);
                tail = sh.npush;
                nh += take_nh();
                spent(3, c0);
            }
        }
        {
            auto id = [&](int k) { return in_win ? sh.win_adj[b0 - wadj0 + k] : ld<CG>(sh.home.g.adj + b0 + k); };
            const int32_t m[1] = {lane < d0 ? id(lane) : (lane == d0 && !self ? s : -1)};
            nh += visit<1, GBM>(t, sh, m, s, cidx, 0, alloc);
            for (int k0 = 32; k0 < d0; k0 += 128) {
                int32_t x[4];
#pragma unroll
                for (int u = 0; u < 4; u++) x[u] = k0 + 32 * u + lane < d0 ? id(k0 + 32 * u + lane) : -1;
                nh += visit<4, GBM>(t, sh, x, s, cidx, 0, alloc);
            }
            if (d0 >= 32 && !self) {   // the row left no lane for s
                const int32_t m1[1] = {lane == 0 ? s : -1};
                nh += visit<1, GBM>(t, sh, m1, s, cidx, 0, alloc);
            }
        }

        // level-synchronous expansion through vertices < s
        int start = 0, end = tail, wstart = 0;
        if (end > 0) {
            const uint32_t c0 = clock32();
            carry(sh, acc, lane);
            __syncwarp();
            do {
                if (end - start <= SOLO_MAX) {
                    __syncwarp();   // the level's queue entries, for every lane
                    n_levels++;
                    nh += expand<CG, GBM>(t, sh, start, end - start, wstart, s, cidx, start, acc, alloc);
                    wstart = start;
                    start = end;
                    end = tail;
                } else {
                    if (lane == 0) {
                        sh.src = s;
                        sh.cidx = cidx;
                        sh.lv_start = start;
                        sh.lv_end = end;
                        sh.lv_wstart = wstart;
                    }
                    collective(OP_LEVELS);
                    start = sh.lv_start;
                    end = sh.lv_end;
                    wstart = sh.lv_wstart;
                    tail = end;
                    nh += take_nh();
                }
            } while (end > start);
            c_levels += since(c0);
        }

        // |hi(s)|: the bits above s; the link flag; both passes' exchange
        hc += nh - 1;
        if (LISTS) total += hc;
        if (nsnap > 0 && end > 0 && lane == 0) {
            sh.weight = min(sh.weight + end, 1 << 28);
            sh.snap_credit = min(sh.snap_credit + end, 1 << 28);
        }
        __syncwarp();
        mine = s + 1 < n && ((t.bits.get((s + 1) >> 5) >> ((s + 1) & 31)) & 1u);
        if (lane == 0) {
            const int64_t slot = sh.home.row + s;
            a.cnt[slot] = hc;
            a.nxt[slot] = mine ? 1 : 0;
        }
        prev = s;
        if (PAIRED) {
            const int par = xch & 1;
            xch++;
            if (lane == 0) pair_flag[par][half] = mine;
            if (nsnap > 0 && lane < SNAP_REACH)
                sh.reach[par][lane] = (s >> 5) + lane < a.bitmap_words ? t.bits.get((s >> 5) + lane) : 0u;
            const uint32_t c0 = clock32();
            pair_sync();
            other = pair_flag[par][1 - half] != 0;
            c_wait += since(c0);
            if (nsnap > 0 && end > 0 && sh.weight >= heavy && sh.snap_credit >= heavy) {
                const long long c0 = clock64();
                int lo, hi;
                state_extent<GBM>(t.bits, lane, lo, hi);
                const int k = sh.snaps & (nsnap - 1);   // nsnap is a power of two
                __syncwarp();
                if (lane < SNAP_REACH) sh.snap_reach[k][lane] = shs[1 - half].reach[par][lane];
                if (lane == 0) {
                    sh.snap_t[k] = s;
                    sh.snaps++;
                    sh.snap_credit -= heavy;
                    sh.snap_w[k] = sh.weight;
                    sh.snap = k;
                    sh.snap_lo[k] = sh.lo = lo;
                    sh.snap_hi[k] = sh.hi = hi;
                }
                collective(OP_SAVE);
                spent(3, c0);
            }
        }
        s += stride;
    }
    fold_work(sh, acc, pass, lane);
    if (lane == 0) {
        const unsigned long long levels = (unsigned long long)c_levels << 8, wait = (unsigned long long)c_wait << 8;
        sh.prof[0] += n_levels;
        sh.prof[2] += levels;
        sh.prof[7] += wait;
        sh.prof[1] += (unsigned long long)clock64() - levels - wait;
        sh.op = OP_EXIT;
    }
    __syncwarp();
    gsync<GT>(bar);
}

// One work piece for a helper thread: the leader's ops until the piece ends.
// Returns the phase of the level counters, which runs on.
template <int BLOCK, bool PAIRED, bool CG, bool GBM, bool LISTS = true>
__device__ __noinline__ int help_piece(Trav<GBM> t, int half, int phase)
{
    using C = CtaOf<BLOCK, PAIRED, LISTS>;
    constexpr int GT = PAIRED ? BLOCK / 2 : BLOCK;
    const int htid = (int)threadIdx.x - half * GT - 32;
    const int bar = 1 + half;
    SharedState &sh = cta<C>().t[half];
    int (*const hist)[32] = cta<C>().hist + (LISTS ? half * (GT / 32 - 1) : 0);
    Tally acc;
    for (;;) {
        gsync<GT>(bar);
        const int op = sh.op;
        if (op == OP_EXIT) break;
        run_op<GT, CG, GBM, LISTS>(cta<C>().a, t, sh, hist, op, htid, bar, phase, acc);
    }
    fold_work(sh, acc, sh.home.pass, htid & 31);
    return phase;
}

// One work piece: the first warp of every traversal leads, the others help.
template <int BLOCK, bool PAIRED, bool CG, bool GBM, bool LISTS = true>
__device__ __forceinline__ void run_piece(const Trav<GBM> &t, int32_t s_lo, int32_t s_hi, int32_t stride, bool shared,
                                          int half, int gtid, int &phase)
{
    if (gtid < 32) {
        __syncwarp();   // the traversal's home, which the first lane has settled
        lead_piece<BLOCK, PAIRED, CG, GBM, LISTS>(t, s_lo, s_hi, stride, shared, half);
    } else {
        phase = help_piece<BLOCK, PAIRED, CG, GBM, LISTS>(t, half, phase);
    }
}

// ---------------------------------------------------------------------------
// The persistent cooperative factorization kernel.
//
// PAIRED = false: every CTA runs one traversal at a time; a work piece is one
// pass of a run of sources, and s reuses s-1's state when s-1 is in adj(s).
// PAIRED = true: the CTA's two halves run pass G and pass G^T of the same
// source side by side, each with its own bitmap and frontier ring, and
// exchange their s+1 flags after every source.  By the fill-path theorem,
// s-1 is in X_G(s) exactly when s is in hi_{G^T}(s-1) (and likewise with G
// and G^T swapped), so each half reuses s-1's state whenever it is valid.
//
// GBM = true: every traversal's visited bitmap and summaries live in global
// memory (a.gbm, resident in L2 for the sizes that matter) instead of shared
// memory, which then holds only the frontier rings: n is bounded only by device
// memory (shared memory holds two bitmaps of at most 844K lines each, 856K for counts).  Two
// CTAs of 512 threads an SM run four traversals side by side; smaller CTAs would
// run more of them, but the one traversal of a whole matrix that a separator
// line needs takes as long as its own helper warps are few (864,008-line
// bordered matrix: 17 ms with seven of them, 39 with three).
//
// MINB: resident CTAs per SM the registers are budgeted for (the default
// fills the SM with 1024 threads; 1 gives a 512-thread CTA up to 128
// registers a thread, for launches that hold one CTA per SM anyway).
// LISTS: the list output is compiled in; counts-only jobs run an
// instantiation without it, whose registers go to the traversal alone.
template <int BLOCK, bool PAIRED, bool GBM, int MINB = (BLOCK >= 1024 ? 1 : 1024 / BLOCK), bool LISTS = true>
__global__ void __launch_bounds__(BLOCK, MINB) factor_kernel(const __grid_constant__ JobArgs a)
{
    constexpr int GT = PAIRED ? BLOCK / 2 : BLOCK;
    constexpr int NS = PAIRED ? 2 : 1;
    using C = CtaOf<BLOCK, PAIRED, LISTS>;
    extern __shared__ __align__(16) uint32_t smem_dyn[];
    C &ca = cta<C>();
    SharedState *const shs = ca.t;
    cg::grid_group grid = cg::this_grid();
    const int tid = threadIdx.x;
    const int half = PAIRED ? tid / GT : 0;
    const int gtid = PAIRED ? tid % GT : tid;
    SharedState &sh = shs[half];
    uint32_t *const smem = smem_dyn + (sizeof(C) + 15) / 16 * 4;
    if (tid == 0) ca.a = a;
    const int64_t trav = (int64_t)blockIdx.x * NS + half;
    uint32_t *const state = GBM ? a.gbm + ((int64_t)blockIdx.x * NS) * a.state_words : smem;
    uint32_t *const ring = (GBM ? smem : smem + (size_t)NS * a.state_words) + (size_t)half * a.ring_size;

    // ---- phase 1: traversals ------------------------------------------------
    unsigned long long t_start = 0;
    if (tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    for (int w = tid; w < NS * a.state_words; w += BLOCK) state[w] = w % a.state_words < STATE_PAD ? ~0u : 0u;
    if (gtid == 0) init_state(sh);
    Trav<GBM> t{};
    t.bits = bits_at<GBM>(state + (size_t)half * a.state_words + STATE_PAD, a.bitmap_words);
    t.f = Frontier{(uint32_t)__cvta_generic_to_shared(ring), a.ring_size};
    if (LISTS && a.want_pattern) t.stamp = a.stamp + trav * (a.stamp_stride + a.stamp_other);
    if (gtid == 0) {
        sh.home.spill = a.queue + trav * a.qcap;
        sh.home.snaps = a.snap + trav * a.snap_k * a.bitmap_words;
        if (LISTS && a.want_pattern) {
            sh.home.stamps = t.stamp;
            sh.home.lists = a.lists + trav * a.qcap;
        }
    }
    int phase = 0, last_mat = -1;
    __syncthreads();
    for (;;) {
        const bool shared = PAIRED && a.shared_piece != nullptr;
        if (tid < 32) {
            long long pc = 0;
            if (tid == 0) pc = (long long)atomicAdd(a.piece_counter, 1ull);
            pc = __shfl_sync(0xffffffffu, pc, 0);
            if (pc >= a.npieces) {
                pc = -1;
                if (shared) {   // no piece is left: a part of another CTA's
                    const unsigned long long w = take_part<C>(gridDim.x, tid);
                    if (tid == 0) ca.word = w;
                }
            }
            if (tid == 0) ca.piece = pc;
        }
        __syncthreads();
        const int64_t pc = ca.piece;
        unsigned long long word = 0ull;
        if (pc < 0) {
            if (!shared) break;
            word = ca.word;
            if (word == 0ull) break;
        }
        int r = 0;
        if (pc < 0) {
            r = (int)(word >> (2 * UNIT_BITS));
        } else {
            int hi = a.nranges - 1;
            while (r < hi) {
                const int mid = (r + hi + 1) >> 1;
                if (a.ranges[mid].piece_base <= pc) r = mid; else hi = mid - 1;
            }
        }
        const Range rg = a.ranges[r];
        const int64_t k = pc - rg.piece_base;
        const int pass = PAIRED ? half : (int)(k & 1);
        int64_t j0, j1;
        if (shared) {
            if (pc >= 0) {   // the range's pieces from its top
                const int units = (rg.nj + UNIT - 1) / UNIT, per = rg.chunk / UNIT;
                const int end = units - (int)k * per;
                word = piece_word(r, end, max(0, end - per));
            }
            j0 = (int64_t)(word & UNIT_MASK) * UNIT;
            if (tid == 0) {   // the first unit is the CTA's own
                SharedPiece &own = shs[0].own;
                own.word = a.shared_piece + blockIdx.x;
                own.cost = a.shared_cost + blockIdx.x;
                own.first = rg.offset;
                own.last = rg.offset + rg.nj;
                own.fresh = a.fresh_cost + fresh_bucket(a.mats[rg.mat].line_base + rg.offset + j0, a.L);
                *reinterpret_cast<volatile unsigned long long *>(own.cost) = 0ull;
                __threadfence();
                atomicExch(own.word, word + 1ull);
            }
            j1 = min(j0 + UNIT, (int64_t)rg.nj);
        } else {
            piece_bounds(rg, PAIRED ? k : (k >> 1), j0, j1);
        }
        const MatDesc md = a.mats[rg.mat];
        const PassGraph g = md.g[pass];
        int32_t s_lo = rg.offset + (int32_t)j0 * rg.stride;
        int32_t s_hi = rg.offset + (int32_t)j1 * rg.stride;   // exclusive (stride 1)
        if (!PAIRED && a.reuse && rg.stride == 1) {
            // cut pieces where adjacency chains start, so a piece's first
            // source rarely has a predecessor it could have reused
            if (tid < 32) {
                const int32_t lim = min(rg.chunk, 64);
                const int32_t lo = (j0 == 0) ? s_lo : chain_start(g, s_lo, lim);
                const int32_t hi = (j1 == rg.nj) ? s_hi : chain_start(g, s_hi, lim);
                if (tid == 0) { sh.seg[0] = lo; sh.seg[1] = hi; }
            }
            __syncthreads();
            s_lo = sh.seg[0];
            s_hi = sh.seg[1];
        }
        if (rg.mat != last_mat && gtid == 0) sh.snap_credit = -1;
        last_mat = rg.mat;
        if (gtid == 0) settle(sh.home, a, md, pass);
        run_piece<BLOCK, PAIRED, false, GBM, LISTS>(t, s_lo, s_hi, rg.stride, shared, half, gtid, phase);
        __syncthreads();   // every thread is done with the piece
    }
    {
        if (tid == 0) {   // this CTA's busy time, summed over CTAs (load balance)
            unsigned long long t_done;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_done));
            atomicAdd(&a.counters[15], t_done - t_start);
        }
        if (tid == 0) {
            unsigned long long ns = 0, nr = 0, wk[3] = {0, 0, 0}, pv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int h = 0; h < NS; h++) {
                for (int q = 0; q < 3; q++) wk[q] += shs[h].work[q] + ((unsigned long long)shs[h].carry[q] << 31);
                ns += shs[h].nsrc;
                nr += shs[h].nsrc - shs[h].nfresh;
                for (int q = 0; q < 8; q++) pv[q] += shs[h].prof[q];
            }
            atomicAdd(&a.counters[0], wk[0]);
            atomicAdd(&a.counters[1], (unsigned long long)ns);
            atomicAdd(&a.counters[3], wk[1]);
            atomicAdd(&a.counters[4], wk[2]);
            atomicAdd(&a.counters[5], (unsigned long long)pv[0]);
            atomicAdd(&a.counters[6], (unsigned long long)nr);
            for (int q = 1; q < 8; q++) atomicAdd(&a.counters[6 + q], (unsigned long long)pv[q]);
        }
    }
    grid.sync();
    if (blockIdx.x == 0 && tid == 0) {   // nanoseconds from launch to the end of the traversals
        unsigned long long t_now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_now));
        a.counters[14] = t_now - t_start;
    }

    const int64_t L = a.L;
    const int64_t ntiles = a.ntiles;

    // line -> matrix lookup (matrices are stored in line order)
    auto mat_of = [&](int64_t l) -> int {
        int lo = 0, hi = a.nmats - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (a.mats[mid].line_base <= l) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    // supernode run boundary before line l: lines l-1 and l join when each
    // is in the other's line and line l's upper count is one less
    auto sn_flag = [&](int64_t l) -> bool {
        const MatDesc &md = a.mats[mat_of(l)];
        const int64_t s = l - md.line_base;
        if (s == 0) return true;
        const bool linked = a.nxt[L + l - 1] && a.nxt[l - 1] && (a.cnt[l] == a.cnt[l - 1] - 1);
        return !linked;
    };

    // ---- phase 2: tile partial sums ------------------------------------------
    for (int64_t t = a.tile_lo + blockIdx.x; t < a.tile_hi; t += gridDim.x) {
        int64_t s0 = 0, s1 = 0, last = -1;
        for (int64_t l = t * TILE + tid; l < min(L, (t + 1) * TILE); l += BLOCK) {
            s0 += a.cnt[l];
            s1 += a.cnt[L + l];
            if (sn_flag(l)) last = max(last, l);
        }
        int64_t t0 = block_sum<BLOCK>(s0, shs[0].warp);
        int64_t t1 = block_sum<BLOCK>(s1, shs[0].warp);
        int64_t tl;
        block_excl_max<BLOCK>(last, &tl, shs[0].warp);
        if (tid == 0) {
            a.tile_sum[t] = t0;
            a.tile_sum[ntiles + t] = t1;
            a.tile_last[t] = tl;
        }
    }
    grid.sync();

    // ---- phase 3: block 0 scans the tile partials -----------------------------
    if (blockIdx.x == 0) {
        int64_t c0 = 0, c1 = 0, cm = -1;
        for (int64_t base = a.tile_lo; base < a.tile_hi; base += BLOCK) {
            const int64_t t = base + tid;
            const int64_t v0 = t < a.tile_hi ? a.tile_sum[t] : 0;
            const int64_t v1 = t < a.tile_hi ? a.tile_sum[ntiles + t] : 0;
            const int64_t vm = t < a.tile_hi ? a.tile_last[t] : -1;
            int64_t tot0, tot1, totm;
            const int64_t e0 = block_excl_scan<BLOCK>(v0, &tot0, shs[0].warp);
            const int64_t e1 = block_excl_scan<BLOCK>(v1, &tot1, shs[0].warp);
            const int64_t em = block_excl_max<BLOCK>(vm, &totm, shs[0].warp);
            if (t < a.tile_hi) {
                a.tile_sum[t] = c0 + e0;
                a.tile_sum[ntiles + t] = c1 + e1;
                a.tile_last[t] = max(cm, em);
            }
            c0 += tot0; c1 += tot1; cm = max(cm, totm);
        }
        if (tid == 0) {
            a.gptr[L] = c0;                  // pass 0 total
            a.gptr[(L + 1) + L] = c1;        // pass 1 total
        }
    }
    grid.sync();

    // ---- phase 4: CSR offsets and supernode starts per tile -------------------
    for (int64_t t = a.tile_lo + blockIdx.x; t < a.tile_hi; t += gridDim.x) {
        int64_t c0 = a.tile_sum[t], c1 = a.tile_sum[ntiles + t], carry = a.tile_last[t];
        int64_t nsn = 0;
        for (int64_t base = t * TILE; base < min(L, (t + 1) * TILE); base += BLOCK) {
            const int64_t l = base + tid;
            const bool in = l < min(L, (t + 1) * TILE);
            int64_t v0 = in ? a.cnt[l] : 0;
            int64_t v1 = in ? a.cnt[L + l] : 0;
            bool f = in && sn_flag(l);
            int64_t tot0, tot1;
            int64_t e0 = block_excl_scan<BLOCK>(v0, &tot0, shs[0].warp);
            int64_t e1 = block_excl_scan<BLOCK>(v1, &tot1, shs[0].warp);
            int64_t sub_last;
            int64_t rs = block_excl_max<BLOCK>(f ? l : -1, &sub_last, shs[0].warp);
            rs = max(max(rs, f ? l : (int64_t)-1), carry);
            bool start = false;
            if (in) {
                a.gptr[l] = c0 + e0;
                a.gptr[(L + 1) + l] = c1 + e1;
                start = f || (a.max_sn > 0 && ((l - rs) % a.max_sn) == 0);
                a.snind[l] = start ? 1 : 0;
            }
            const int64_t ns = block_sum<BLOCK>(start ? 1 : 0, shs[0].warp);
            carry = max(carry, sub_last);   // run start carried to the next sub-tile
            c0 += tot0; c1 += tot1; nsn += ns;
        }
        if (tid == 0) a.tile_sn[t] = nsn;
    }
    grid.sync();

    // ---- phase 5: block 0 scans the supernode tile counts ---------------------
    if (blockIdx.x == 0) {
        int64_t c = 0;
        for (int64_t base = a.tile_lo; base < a.tile_hi; base += BLOCK) {
            const int64_t t = base + tid;
            int64_t v = t < a.tile_hi ? a.tile_sn[t] : 0;
            int64_t tot;
            int64_t e = block_excl_scan<BLOCK>(v, &tot, shs[0].warp);
            if (t < a.tile_hi) a.tile_sn[t] = c + e;
            c += tot;
        }
        if (tid == 0) a.counters[2] = (unsigned long long)c;
    }
    grid.sync();

    // ---- phase 6: supernode list, pattern compaction ---------------------------
    for (int64_t t = a.tile_lo + blockIdx.x; t < a.tile_hi; t += gridDim.x) {
        int64_t c = a.tile_sn[t];
        for (int64_t base = t * TILE; base < min(L, (t + 1) * TILE); base += BLOCK) {
            const int64_t l = base + tid;
            const bool in = l < min(L, (t + 1) * TILE);
            int64_t v = (in && a.snind[l]) ? 1 : 0;
            int64_t tot;
            int64_t e = block_excl_scan<BLOCK>(v, &tot, shs[0].warp);
            if (v) a.sn_list[c + e] = (int32_t)l;
            if (in && a.mat_info) {
                const int mi = mat_of(l);
                if (a.mats[mi].line_base == l) {
                    a.mat_info[3 * mi + 0] = a.gptr[l];
                    a.mat_info[3 * mi + 1] = a.gptr[(L + 1) + l];
                    a.mat_info[3 * mi + 2] = c + e;
                }
            }
            c += tot;
        }
    }
    // CSR form only (want_pattern == 1); the ranges form (2) leaves the
    // lists where the chains wrote them, at poff
    if (a.want_pattern == 1 && (*a.status & ERR_POOL_OVERFLOW) == 0) {
        const int warps = (gridDim.x * BLOCK) >> 5;
        const int gw = (blockIdx.x * BLOCK + tid) >> 5;
        const int lane = tid & 31;
        const int64_t tot0 = a.gptr[L];
        for (int64_t pl = gw; pl < 2 * L; pl += warps) {
            const int pass = pl >= L;
            const int64_t l = pass ? pl - L : pl;
            const int32_t c = a.cnt[pl];
            if (c == 0) continue;
            const int64_t src = a.poff[pl];
            const int64_t dst = (pass ? tot0 : 0) + a.gptr[pass * (L + 1) + l];
            // four loads in flight per lane before their stores
            const int32_t *from = a.pool + src;
            int32_t *to = a.out + dst;
            for (int32_t k0 = 0; k0 < c; k0 += 128) {
                int32_t v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int32_t k = k0 + 32 * u + lane;
                    v[u] = k < c ? __ldcs(from + k) : 0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int32_t k = k0 + 32 * u + lane;
                    if (k < c) __stcs(to + k, v[u]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Upload kernels: validation, diagonal removal, distinct-entry counts, G^T.

struct UploadArgs {
    int32_t n;
    int64_t nnz;
    const int32_t *beg, *end, *adj;  // staged input
    int32_t *deg;                    // [n]   distinct off-diagonal entries per line
    int32_t *indeg;                  // [n+1] entries per transposed line
    int32_t *orig_up;                // [n]   distinct entries > v in line v
    int32_t *orig_lo;                // [n]   distinct lines u > j holding j
    int32_t *rawdeg;                 // [n]   end[v] - beg[v]
    unsigned long long *counts;      // [0] distinct upper, [1] distinct lower
    uint32_t *status;                // bit 0: invalid input
};

// True when adj[k] is the first occurrence of its value in line [b, k].
__device__ __forceinline__ bool first_in_line(const int32_t *adj, int32_t b, int32_t k,
                                              bool sorted)
{
    const int32_t m = adj[k];
    if (sorted) return (k == b) || (adj[k - 1] != m);
    for (int32_t j = b; j < k; j++)
        if (adj[j] == m) return false;
    return true;
}

// One warp per line.  Checks the range and the ids, counts kept entries and
// transposed entries, and the distinct off-diagonal entries above/below.
__global__ void upload_count_kernel(UploadArgs u)
{
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long up = 0, lo = 0;
    for (int64_t v = gw; v < u.n; v += nw) {
        const int32_t b = u.beg[v], e = u.end[v];
        if (b < 0 || e < b || (int64_t)e > u.nnz) {
            if (lane == 0) {
                atomicOr(u.status, 1u);
                u.deg[v] = 0; u.orig_up[v] = 0; u.rawdeg[v] = 0;
            }
            continue;
        }
        if (lane == 0) u.rawdeg[v] = e - b;
        // sorted lists allow a linear duplicate test
        bool sorted = true;
        for (int32_t k = b + lane; k + 1 < e; k += 32)
            if (u.adj[k] > u.adj[k + 1]) sorted = false;
        sorted = __all_sync(0xffffffffu, sorted);
        int kept = 0, kup = 0;
        for (int32_t k = b + lane; k < e; k += 32) {
            const int32_t m = u.adj[k];
            if (m < 0 || m >= u.n) { atomicOr(u.status, 1u); continue; }
            if (m == (int32_t)v) continue;
            if (!first_in_line(u.adj, b, k, sorted)) continue;
            kept++;
            atomicAdd(&u.indeg[m], 1);
            if (m > v) { up++; kup++; }
            else { lo++; atomicAdd(&u.orig_lo[m], 1); }
        }
        for (int o = 16; o; o >>= 1) {
            kept += __shfl_xor_sync(0xffffffffu, kept, o);
            kup += __shfl_xor_sync(0xffffffffu, kup, o);
        }
        if (lane == 0) { u.deg[v] = kept; u.orig_up[v] = kup; }
    }
    for (int o = 16; o; o >>= 1) {
        up += __shfl_xor_sync(0xffffffffu, up, o);
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
    }
    if (lane == 0) {
        if (up) atomicAdd(&u.counts[0], up);
        if (lo) atomicAdd(&u.counts[1], lo);
    }
}

// One warp per line: copies the kept entries (order preserved) into G and
// scatters them into G^T through per-line cursors.
__global__ void upload_fill_kernel(UploadArgs u, const int32_t *gptr, int32_t *gadj,
                                   int32_t *tcursor, int32_t *tadj)
{
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = gw; v < u.n; v += nw) {
        const int32_t b = u.beg[v], e = u.end[v];
        if (b < 0 || e < b || (int64_t)e > u.nnz) continue;
        bool sorted = true;
        for (int32_t k = b + lane; k + 1 < e; k += 32)
            if (u.adj[k] > u.adj[k + 1]) sorted = false;
        sorted = __all_sync(0xffffffffu, sorted);
        int32_t out = gptr[v];
        for (int32_t k0 = b; k0 < e; k0 += 32) {
            const int32_t k = k0 + lane;
            int32_t m = -1;
            bool keep = false;
            if (k < e) {
                m = u.adj[k];
                keep = (m >= 0 && m < u.n && m != (int32_t)v) &&
                       first_in_line(u.adj, b, k, sorted);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                gadj[out + __popc(bal & ((1u << lane) - 1u))] = m;
                const int32_t p = atomicAdd(&tcursor[m], 1);
                tadj[p] = (int32_t)v;
            }
            out += __popc(bal);
        }
    }
}

// Fills the 32-byte slot of every vertex of one pass graph: {degree, input
// degree (pass G) or, of rows longer than SLOT_NB, the row's offset, the first
// SLOT_NB ids (-1 past the degree)}; one empty slot follows the last.
__global__ void slot_fill_kernel(int32_t n, const int32_t *ptr, const int32_t *adj, const int32_t *rawdeg, int4 *slot)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (int64_t)gridDim.x * blockDim.x) {
        if (v == n) {
            slot[2 * v] = make_int4(0, 0, -1, -1);
            slot[2 * v + 1] = make_int4(-1, -1, -1, -1);
            break;
        }
        const int32_t b = ptr[v], d = ptr[v + 1] - b;
        int32_t x[SLOT_NB];
#pragma unroll
        for (int u = 0; u < SLOT_NB; u++) x[u] = u < d ? adj[b + u] : -1;
        slot[2 * v] = make_int4(d, d > SLOT_NB ? b : (rawdeg ? rawdeg[v] : 0), x[0], x[1]);
        slot[2 * v + 1] = make_int4(x[2], x[3], x[4], x[5]);
    }
}

// Exclusive scan of int32 counts into int32 offsets: three kernels.
template <int BLOCK>
__global__ void scan_tiles_kernel(const int32_t *in, int64_t n, int64_t *tile_sums)
{
    __shared__ int64_t warp[32];
    const int64_t t = blockIdx.x;
    const int64_t i = t * BLOCK + threadIdx.x;
    int64_t v = i < n ? in[i] : 0;
    int64_t s = block_sum<BLOCK>(v, warp);
    if (threadIdx.x == 0) tile_sums[t] = s;
}

template <int BLOCK>
__global__ void scan_partials_kernel(int64_t *tile_sums, int64_t ntiles, int64_t *total)
{
    __shared__ int64_t warp[32];
    int64_t c = 0;
    for (int64_t base = 0; base < ntiles; base += BLOCK) {
        const int64_t t = base + threadIdx.x;
        int64_t v = t < ntiles ? tile_sums[t] : 0;
        int64_t tot;
        int64_t e = block_excl_scan<BLOCK>(v, &tot, warp);
        if (t < ntiles) tile_sums[t] = c + e;
        c += tot;
    }
    if (threadIdx.x == 0) *total = c;
}

template <int BLOCK>
__global__ void scan_apply_kernel(const int32_t *in, int64_t n, const int64_t *tile_sums,
                                  int32_t *out, const int64_t *total)
{
    __shared__ int64_t warp[32];
    const int64_t t = blockIdx.x;
    const int64_t i = t * BLOCK + threadIdx.x;
    int64_t v = i < n ? in[i] : 0;
    int64_t tot;
    int64_t e = block_excl_scan<BLOCK>(v, &tot, warp);
    if (i < n) out[i] = (int32_t)(tile_sums[t] + e);
    if (i == 0) out[n] = (int32_t)*total;
}

}  // namespace dev
}  // namespace gsofa
