// Shared host/device definitions of the GB300 BiWFA engine.
//
// Layout in HBM for one batch (all device buffers are owned by a wfg_context_t):
//   seq_ascii   : the batch's raw pattern/text bytes, concatenated (uploaded once per batch)
//   seq_words   : per pair, four packed arrays [P fwd | T fwd | P rev | T rev], each
//                 ceil(len*bits/32)+2 uint32 words (2 zero pad words so a 64-bit window
//                 read never leaves the array). bits = 2 for pure ACGT pairs, else 8.
//   arena       : one private scratch slab per resident warp (rings, leaf store, runs, stack)
//   out_runs    : dense CIGAR output, uint32 (len<<4 | op) SAM-style ops, one contiguous
//                 span per pair reserved with one atomicAdd when the pair finishes
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define WFG_HD __host__ __device__
#else
#define WFG_HD
#endif

#ifdef __cplusplus
namespace wfg {
#endif

// SAM BAM op codes used in the output runs (op '=' is a match, 'X' a mismatch).
enum { WFG_OP_INS = 1, WFG_OP_DEL = 2, WFG_OP_EQ = 7, WFG_OP_X = 8 };

// Internal per-pair statuses beyond WFA2's public ones.
enum {
  WFG_ST_COMPLETED = 0,
  WFG_ST_MAX_STEPS = -100,
  WFG_ST_OOM = -200,              // WFA2's WF_STATUS_OOM
  WFG_ST_UNATTAINABLE = -300,
  WFG_ST_SCRATCH_OVERFLOW = -210, // the pair needs a larger per-warp arena (retried by the host)
  WFG_ST_DEVICE_ERROR = -500,     // WF_STATUS_DEVICE_ERROR
  WFG_ST_OUTPUT_OVERFLOW = -220,  // the dense output span could not be reserved
};

struct PairDesc {
  int64_t word_off;   // first word of this pair's packed arrays in seq_words
  int64_t p_off;      // pattern / text byte offsets in seq_ascii
  int64_t t_off;
  int plen, tlen;
  int pw_len, tw_len; // words per packed pattern / text array (incl. 2 pad words)
  int bits;           // 2 or 8 (set by the pack kernel)
  int pad;
};

struct KernelParams {
  // penalties: internal (transformed when match < 0) and the caller's for rescoring
  int x, o, e, scope;
  int o2, e2;                // second gap piece (two-piece gap-affine), internal
  int match_o, x_o, o_o, e_o;
  int o2_o, e2_o;            // second gap piece as the caller gave it
  int metric;                // 0 gap-affine, 1 edit, 2 indel, 3 gap-linear, 4 two-piece gap-affine
                             // (x, o, e, scope already set for it)
  int score_only;
  int max_steps;
  // pairs
  int num_pairs;             // used when num_pairs_ptr is null
  const unsigned long long* num_pairs_ptr; // device count (retry passes read the previous pass's count)
  const PairDesc* pairs;
  const int* order;          // processing order (work-stealing queue)
  int* retry_out;            // pairs that overflowed the arena are appended here (null: final pass)
  unsigned long long* retry_count;  // append cursor of retry_out
  unsigned long long* queue_head;   // work-queue cursor of this pass
  const uint32_t* words;
  // per-warp arena
  uint8_t* arena;
  int64_t arena_bytes;       // bytes per warp
  int ring_w;                // ring width (power of two, diagonals per wavefront slot)
  int leaf_words;            // int32 capacity of the leaf wavefront store
  int leaf_max_score;        // capacity of the leaf descriptor table (scores)
  int run_cap;               // uint32 capacity of the per-pair run list
  int leaf_run_cap;          // uint32 capacity of the leaf reverse-run buffer
  int stack_cap;             // recursion stack entries
  // outputs
  int* scores;
  int* status;
  int64_t* run_off;
  int* run_len;
  uint32_t* out_runs;
  int64_t out_cap;
  unsigned long long* out_head;  // dense output cursor (shared by all passes)
  // statistics (optional, may be null; not from the tile kernel): per pair {n_steps, max_leaf_score, max_depth, n_cells}
  int* stats;
  // execution shape (0 = defaults): warps cooperating on one pair, rings in shared memory,
  // physical ring buffers per direction (<= scope; see ring_buffers())
  int group_warps;
  int ring_in_smem;
  int ring_nphys;
  // rows in tiles (biwfa_tiles.cuh): the spacing of the scores that hold a row, 0 for one score at a time
  int tile_g;
  int tile_owners;  // and the warps of a block that own pairs
  // the tile kernel's waits for another warp: counter of those that ran out (the run has failed then),
  // and their limit in polls (0: from the pair's length)
  unsigned long long* lost;
  int wait_polls;
};

// Score scope caps (max(x, o+e[, o2+e2]) + 1 after the match transform): the ring descriptors
// live in shared memory, sized for the cap of each kernel instantiation (32 for the usual
// penalties; 64 for larger ones and for two-piece gap-affine).
#define WFG_MAX_SCOPE 32
#define WFG_MAX_SCOPE_2P 64

// Rows in tiles: ring buffers per direction, ints between the end of a ring row and the next (a
// pitch that is no power of two spreads the rows over the caches' sets), and the diagonals beyond
// a pair's own that a ring row must hold (the last tile's unused lanes and the halos).
#define WFG_TILE_BUFS 12
#define WFG_TILE_PAD 64
#define WFG_TILE_MARGIN 160
// Null offset of the tile kernel's rows (biwfa_tiles.cuh), between two bounds: below minus 17 for each
// row of a search (2^25 + scope), and twice it less a diagonal (2^27) within 32 bits.
#define WFG_TILE_NULL (-(5 << 27))
static_assert(WFG_TILE_NULL + 17 * ((int64_t)(1 << 25) + 2 * WFG_MAX_SCOPE) < 0, "a null stays negative");
static_assert(2 * (int64_t)WFG_TILE_NULL - (1 << 27) - 8 >= INT32_MIN, "twice a null fits 32 bits");

// Ints from the start of a direction's tile rings to row `row` (buffer * 3 + component). 64 bits: the
// longest accepted pairs (plen + tlen just below 2^26, at unit penalties) have rings of 2^27 diagonals,
// and the last of 36 rows starts beyond 2^31 ints from 2^26 diagonals on. Within a block's 12 rows
// 32 bits do.
WFG_HD constexpr inline int64_t wfg_tile_row(int row, int pitch) { return (int64_t)row * pitch; }
static_assert(12 * (int64_t)((1 << 27) + WFG_TILE_PAD) <= INT32_MAX, "a block's rows are indexed with 32 bits");

// The leaf store of a leaf whose rows come in tiles: row 0's one cell at 0, then block b's four rows
// (rows 4b + 1 .. 4b + 4; M, I and D each, or M alone), all of one size, from wfg_tile_leaf_at(b), all
// multiples of 4. Gap-affine rows span at most t diagonals on either side, 8b + 8 in all with one side
// shorter by the gap opening; one-component rows t / lo on each side (lo: rows back to the gap source),
// so with q = b / lo they lie within 4q + 4 of the middle. q = b for gap-affine.
WFG_HD constexpr inline int wfg_tile_leaf_n(bool linear, int q) { return linear ? 8 * q + 12 : 8 * q + 8; }
WFG_HD constexpr inline int wfg_tile_leaf_at(bool linear, int b, int q, int lo) {
  // one component: 4 rows x sum over i < b of (8 (i / lo) + 12)
  return 4 + (linear ? 48 * b + 16 * q * (2 * b - lo * (q + 1)) : 48 * b * (b + 1));
}

// Words of a leaf store that holds every row of a leaf up to score smax, in a batch whose longest pair
// has plen + tlen = maxsum; g: the spacing of the scores with a row. One score at a time a step at score
// s takes at most ncomp * min(maxsum + 8, 2 s / emin + 8). Rows in tiles are not clipped to the window, so
// where they need more, up to the largest score of a leaf (reach), that counts, and a last block's rows
// beyond it.
WFG_HD constexpr inline int64_t wfg_leaf_words(int smax, int maxsum, int g, int emin, int ncomp, bool tiles, bool linear,
                                               int lo, int64_t reach) {
  int64_t w = 0, tile = 0;
  int q = 0, next = 4 * lo;  // q = (t - 1) / (4 lo) of row t = s / g
  for (int s = 0, t = 0; s <= smax; s += g, ++t) {
    const int64_t step = 2LL * s / emin + 8, clip = maxsum + 8;
    int64_t row = ncomp * (step < clip ? step : clip);
    if (tiles && s <= reach) {
      if (t > next) { ++q; next += 4 * lo; }
      tile = (int64_t)(linear ? 1 : 3) * wfg_tile_leaf_n(linear, q);
      if (tile > row) row = tile;
    }
    w += row;
  }
  return w + 4 * tile;
}

// Physical ring buffers a direction needs: scores that can hold a wavefront are multiples of
// g = gcd(x, o+e, e), so any window of `scope` consecutive scores holds at most ceil(scope/g)
// live wavefronts, and round-robin buffers of that count are never overwritten while needed.
WFG_HD constexpr inline int wfg_gcd(int a, int b) { return b == 0 ? a : wfg_gcd(b, a % b); }
WFG_HD constexpr inline int wfg_ring_buffers(int x, int o, int e) {
  return ((o + e > x ? o + e : x) + 1 + wfg_gcd(wfg_gcd(x, o + e), e) - 1) / wfg_gcd(wfg_gcd(x, o + e), e);
}
// The same for two gap pieces: g = gcd(x, o1+e1, e1, o2+e2, e2) over scope = max(x, o1+e1,
// o2+e2) + 1.
WFG_HD constexpr inline int wfg_ring_buffers_2p(int x, int o1, int e1, int o2, int e2) {
  return ((o1 + e1 > x ? (o1 + e1 > o2 + e2 ? o1 + e1 : o2 + e2) : (x > o2 + e2 ? x : o2 + e2)) + 1 +
          wfg_gcd(wfg_gcd(wfg_gcd(x, o1 + e1), wfg_gcd(e1, o2 + e2)), e2) - 1) /
         wfg_gcd(wfg_gcd(wfg_gcd(x, o1 + e1), wfg_gcd(e1, o2 + e2)), e2);
}

// Per-warp arena carving (bytes); all offsets 256-byte aligned.
struct ArenaLayout {
  int64_t ring_off, ring_bytes;     // 2 directions x buffers x ncomp components x ring_w int32
  int64_t ldesc_off, ldesc_bytes;   // (leaf_max_score+1) x ncomp x int4
  int64_t ldata_off, ldata_bytes;   // leaf_words int32
  int64_t runs_off, runs_bytes;     // run_cap uint32
  int64_t lruns_off, lruns_bytes;   // leaf_run_cap uint32
  int64_t stack_off, stack_bytes;   // stack_cap x 8 int32
  int64_t rdesc2_off, rdesc2_bytes; // I2/D2 ring descriptors, 2 directions x WFG_MAX_SCOPE_2P
                                    // scores x 2 x int2 (ncomp == 5 only)
  int64_t total;
};

WFG_HD constexpr inline int64_t wfg_align256(int64_t v) { return (v + 255) & ~(int64_t)255; }

// ncomp: 3 (M, I1, D1) or 5 (two-piece gap-affine: + I2, D2).
WFG_HD constexpr inline ArenaLayout wfg_arena_layout(int scope, int ring_w, int leaf_max_score, int leaf_words,
                                           int run_cap, int leaf_run_cap, int stack_cap, int ncomp = 3) {
  ArenaLayout L{};
  int64_t off = 0;
  L.ring_off = off; L.ring_bytes = wfg_align256((int64_t)2 * scope * ncomp * ring_w * 4); off += L.ring_bytes;
  L.ldesc_off = off; L.ldesc_bytes = wfg_align256((int64_t)(leaf_max_score + 1) * ncomp * 16); off += L.ldesc_bytes;
  L.ldata_off = off; L.ldata_bytes = wfg_align256((int64_t)leaf_words * 4); off += L.ldata_bytes;
  L.runs_off = off; L.runs_bytes = wfg_align256((int64_t)run_cap * 4); off += L.runs_bytes;
  L.lruns_off = off; L.lruns_bytes = wfg_align256((int64_t)leaf_run_cap * 4); off += L.lruns_bytes;
  L.stack_off = off; L.stack_bytes = wfg_align256((int64_t)stack_cap * 8 * 4); off += L.stack_bytes;
  L.rdesc2_off = off;
  L.rdesc2_bytes = ncomp == 5 ? wfg_align256((int64_t)2 * WFG_MAX_SCOPE_2P * 2 * 8) : 0;
  off += L.rdesc2_bytes;
  L.total = off;
  return L;
}

#ifdef __cplusplus
}  // namespace wfg
#endif
