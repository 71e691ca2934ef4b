// The kernel whose wavefront rows come in tiles (biwfa_tiles.cuh): score + CIGAR for gap-affine
// penalties with x = 2g, o+e = 4g, e = g and for the one-component distances. Included by biwfa_kernel.cu inside namespace wfg.
//
// A warp owns a pair. Its work is a loop of blocks (four rows of one or both directions); the code
// that computes a block stands once, in the kernel's loop, with the two common continuations (the
// next block of a breakpoint search without an event, the next block of a leaf) behind it.
// Everything else — the queue, the recursion, the second phase of a search, backtraces, output — is
// tile_control(), called when the common continuation does not apply; it runs on the state in
// shared memory until it needs another block. So the block's code is neither duplicated nor called:
// registers saved around calls and instructions fetched for copies cost as much as 15 % (150,000
// mixture pairs, same GB300: 213-219 ms with two levels of calls per block, 180-191 ms with one).
//
// Warps of a thread block whose queue has run dry compute tiles of the block's other warps (jobs,
// below): the longest pairs of a batch, or the few pairs of a small one, would otherwise take as long
// as one warp needs for them.

namespace {

// One thread block of 16 warps per SM (128 registers a thread): a pair at the end of a batch then has
// up to 15 helpers. Measured end to end on a GB300, one block of 16 / two of 10 / four of 5 warps:
// one 10 kbp pair 8.6 / 9.9 / 11.8 ms, 48 pairs of 10-20 kbp 124 / 156 / 237 ms, 20,000 uneven pairs
// 72.7 / 76.1 / 84.5 ms, 150,000 mixture pairs 171 / 177 / 188 ms, 10,000 pairs of 1 kbp 3.38 / 3.56 /
// 3.58 ms, 200,000 of 150 bp 12.5 / 12.4 / 12.8 ms. Without helpers (a warp per block, 20 an SM):
// 21.5, 122 (eight warps a pair), 101, 182, 3.79, 13.4 ms.
#ifndef WFG_TILE_WARPS
#define WFG_TILE_WARPS 16
#endif
#ifndef WFG_TILE_BLOCKS
#define WFG_TILE_BLOCKS 1
#endif
constexpr int kTileWarps = WFG_TILE_WARPS;    // warps per thread block
constexpr int kTileBlocks = WFG_TILE_BLOCKS;  // thread blocks per SM
// Limits of the waits for other warps, in polls. A poll costs 20 ns at least. A tile ends by itself; the
// longest follow four diagonals over both whole sequences, at worst half a window (4 bases of 8 bits) per
// base and 1 us of memory latency per window, so an owner polls 128 times per base of its pair beyond
// the constant before it gives a helper up. A helper without work leaves after about 10 s.
constexpr int kSpinLimit = 1 << 24, kPollsPerBase = 128;
// Most warps of a block that own pairs, by the launch's warps per pair; the others help. A launch of
// few pairs has fewer owners (KernelParams::tile_owners), each of which needs an arena.
__host__ __device__ constexpr int biwfa_owners(int group_warps) {
  return group_warps <= 1 ? kTileWarps : group_warps == 4 ? 2 : 1;
}

// What a warp is doing between two blocks.
enum { kFetch, kSearch, kSearchEvent, kMeet, kLeaf, kLeafEvent, kHelp, kOwnJob };
// Which tiles a block pass covers: one direction, one tile of each direction in half a warp, both.
enum { kOne, kHalves, kBoth };

// A block that its owner shares with the thread block's idle warps. The ticket word holds
// {generation, tiles, next tile}: a warp takes a tile with one add, and since the generation and the
// number of tiles come back with the tile's number, a late add to a job that has ended takes nothing.
// The fields hold until all tiles are done, so they are read after a tile is taken.
struct TileJob {
  unsigned long long ticket;  // generation << 48 | tiles << 24 | next tile
  int done;                   // tiles computed
  int t0, d_tiles, tiles;     // tiles 0 .. d_tiles - 1 are dir[d]'s, the rest dir[1]'s
  int d;
  int part[10];               // results: d's antidiagonals of four rows and first touched row, then e's
};

// A group's arena (csrc/wfg_internal.h).
struct TileArena { int4* ldesc; int32_t* ldata; uint32_t* runs; uint32_t* lruns; int* stack; int32_t* ring; };

// A warp's state between blocks, in shared memory.
struct TileCtl {
  int state;
  int mode, d, t0, tile, step;  // the block to compute: dir[d] (and dir[1]), tiles tile, tile + step, ...
  int owner;                    // the warp whose directions these are
  bool second;                  // the tile belongs to the second direction of a job
  int after;                    // state that follows an own job
  int part[10];                 // results of the block, as TileJob's
  // pair
  bool first;
  int pi, status, score, sp;
  PairSeqs q;
  RunOut out;
  // window
  int pb, pe, tb, te, cb, ce, rem;
  // search
  int guard, max_antidiag, fmax, rmax, sf, sr;
  bool last_fwd;
  BP bp;
  // leaf
  int leaf_end;  // words of the leaf store in use
};

struct TileGroup {
  Dir dir[3];  // F, R, B
  int2 rdesc[2][kMaxScope * 3];
  int rphys[2][kMaxScope];
  Pen pen;
  TileArena arena;
  TileCtl ctl;
  TileJob job;
};

struct TileBlockSmem {
  TileGroup grp[kTileWarps];
  KernelParams P;
  int active, idle;  // warps with a pair, warps that help
};
// The block's shared memory, named rather than passed: a function that gets a pointer to it reads it
// with generic loads and 64-bit addresses, a third more code.
static_assert(sizeof(TileBlockSmem) <= 48 * 1024, "more shared memory than a launch gets without asking");
extern __shared__ __align__(16) unsigned char s_tile_smem[];
__device__ __forceinline__ TileBlockSmem& tile_smem() { return *reinterpret_cast<TileBlockSmem*>(s_tile_smem); }

__device__ __forceinline__ int job_next(unsigned long long ticket) { return (int)(ticket & 0xffffffu); }
__device__ __forceinline__ int job_tiles(unsigned long long ticket) { return (int)((ticket >> 24) & 0xffffffu); }

// A word that other warps write while this one decides by it: one lane reads it for all, as lanes
// that read it one after another could decide differently and part at the next shuffle.
__device__ __forceinline__ int warp_read(const int& word, int lane) {
  return __shfl_sync(kFull, lane == 0 ? *(const volatile int*)&word : 0, 0);
}

// Takes a tile of the job for this warp: its number, or -1.
__device__ __forceinline__ int job_take(TileJob& job, int lane) {
  int i = -1;
  if (lane == 0) {
    const unsigned long long seen = *(volatile unsigned long long*)&job.ticket;
    if (job_next(seen) < job_tiles(seen)) {
      const unsigned long long got = atomicAdd(&job.ticket, 1ull);
      if (job_next(got) < job_tiles(got)) i = job_next(got);
    }
  }
  i = __shfl_sync(kFull, i, 0);
  if (i >= 0) { __threadfence_block(); __syncwarp(); }
  return i;
}

// Sets the block pass of tile i of the job of warp `owner`.
__device__ __forceinline__ void job_block(int owner, int i, TileCtl& C) {
  const TileJob& job = tile_smem().grp[owner].job;
  C.owner = owner;
  C.mode = kOne;
  C.second = i >= job.d_tiles;
  C.d = C.second ? 1 : job.d;
  C.t0 = job.t0;
  C.tile = i < job.d_tiles ? i : i - job.d_tiles;
  C.step = 1 << 24;
}

// Adds the results of a tile (C.part) to its job.
__device__ __forceinline__ void job_add(const TileCtl& C, int lane) {
  TileJob& job = tile_smem().grp[C.owner].job;
  int* out = job.part + (C.second ? 5 : 0);
  if (lane < 4) atomicMax(&out[lane], C.part[lane]);
  if (lane == 4) atomicMin(&out[4], C.part[4]);
  __threadfence_block();
  __syncwarp();
  if (lane == 0) atomicAdd(&job.done, 1);
}

// The state of direction d after block t0: touch is its first touched row of the four, 4 if none.
__device__ __forceinline__ void tile_done(Dir& d, int t0, int touch) {
  d.ts.lo = d.ts.base;
  d.ts.hi = d.ts.end;
  d.ts.t = t0 + 4;
  d.ts.touched = touch < 4 ? 1 : 0;
  d.ts.valid = touch < 4 ? t0 + 1 + touch : t0 + 4;
}

// Opens block t0 of dir[d] (both: and of dir[1]), more than one tile, to the thread block's idle warps
// and takes a tile of it as this warp's next pass. state: what follows the job.
__device__ __noinline__ void job_open(int d, bool both, int t0, int state, int gib, int lane) {
  TileGroup& S = tile_smem().grp[gib];
  TileCtl& C = S.ctl;
  TileJob& job = S.job;
  const int nd = S.dir[d].ts.tiles, tiles = nd + (both ? S.dir[1].ts.tiles : 0);
  if (lane < 10) job.part[lane] = lane == 4 || lane == 9 ? 4 : INT_MIN;
  if (lane == 0) { job.d = d; job.d_tiles = nd; job.tiles = tiles; job.t0 = t0; job.done = 0; }
  __syncwarp();
  if (lane == 0) {
    __threadfence_block();
    const unsigned long long gen = (*(volatile unsigned long long*)&job.ticket >> 48) + 1;
    atomicExch(&job.ticket, (gen << 48) | ((unsigned long long)tiles << 24));
  }
  __syncwarp();
  C.after = state;
  C.state = kOwnJob;
  const int i = job_take(job, lane);
  if (i >= 0) job_block(gib, i, C);
  else C.step = 0;  // the helpers took every tile: nothing to compute here
  __syncwarp();
}

// Sets up block t0 of dir[d] (both: and of dir[1]) as the warp's next pass, alone or as a job that
// the block's idle warps share. state: what follows it. False when a ring does not hold the block.
template <bool LIN>
__device__ __noinline__ bool tile_request(int d, bool both, int t0, int state, int gib, int lane) {
  TileBlockSmem& B = tile_smem();
  TileGroup& S = B.grp[gib];
  TileCtl& C = S.ctl;
  const bool halves = both && tile_half<LIN>(S.dir[0].cb, t0, S.pen) && tile_half<LIN>(S.dir[1].cb, t0, S.pen);
  const int L = halves ? 16 : 32;
  if (!tile_plan<LIN>(S.dir[d], t0, L, S.pen) || (both && !tile_plan<LIN>(S.dir[1], t0, L, S.pen))) return false;
  if (halves && !(S.dir[0].ts.narrow && S.dir[1].ts.narrow)) {  // one width for both
    S.dir[0].ts.narrow = S.dir[1].ts.narrow = 0;
    S.dir[0].ts.end = S.dir[0].ts.base + 64;
    S.dir[1].ts.end = S.dir[1].ts.base + 64;
  }
  C.owner = gib; C.d = d; C.t0 = t0; C.tile = 0; C.step = 1;
  if (!LIN) {  // which rows' I and D go to the ring (TileArgs::gaps)
    S.dir[d].ts.gaps = state == kMeet || (state == kSearch && S.dir[d].ts.tiles <= kGapTiles);
    if (both) S.dir[1].ts.gaps = S.dir[1].ts.tiles <= kGapTiles;
  }
  C.state = state;
  C.mode = halves ? kHalves : both ? kBoth : kOne;
  __syncwarp();
  if (!halves && state != kLeaf && S.dir[d].ts.tiles + (both ? S.dir[1].ts.tiles : 0) > 1 && warp_read(B.idle, lane) > 0)
    job_open(d, both, t0, state, gib, lane);
  return true;
}

// I and D of the last two blocks of both directions of a search, where their passes did not store them.
__device__ __noinline__ void search_gaps(int gib, int lane) {
  TileGroup& S = tile_smem().grp[gib];
  #pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int t0 = S.ctl.t0 - (i < 2 ? 4 : 0);
    if (t0 >= 0 && tile_wide(S.dir[i & 1].cb, t0, S.pen)) tile_gaps(S.dir[i & 1], t0, S.pen, lane);
  }
}

// Runs the warp's state machine to its next block pass (S.ctl says which); false when the launch has
// no more work for this warp.
template <bool LIN>
__device__ __noinline__ bool tile_control(int gib, int lane, int owners) {
  TileBlockSmem& B = tile_smem();
  TileGroup& S = B.grp[gib];
  TileCtl& C = S.ctl;
  const KernelParams& P = B.P;
  Dir& F = S.dir[0];
  Dir& R = S.dir[1];
  Dir& L = S.dir[2];
  const Pen& pen = S.pen;
  Grp<1> g;
  g.tid = lane; g.bar = 0; g.red = nullptr;
  enum { kPop = 100, kMet, kSteps, kBpDone, kLeafSteps, kFinish };
  int state = C.state, st = ST_OK, resume = 0;
  RunOut out = C.out;
  BP bp = C.bp;
  bool done = false, resumed = false;
  int s = 0;

  if (state == kHelp || state == kOwnJob) {
    if (state == kOwnJob) {  // no tile is left to take: wait for the helpers'
      const int tiles = S.job.tiles;
      const long long limit = P.wait_polls > 0 ? P.wait_polls
                                               : kSpinLimit + (long long)kPollsPerBase * (C.q.plen + C.q.tlen);
      long long polls = 0;
      bool ended;
      while (!(ended = warp_read(S.job.done, lane) >= tiles) && polls < limit) { ++polls; __nanosleep(20); }
      if (!ended) {
        // A helper holds a tile of this warp's rings and job, now or later: nothing may use them again in
        // this launch. The run has failed; the warp takes no more pairs.
        if (lane == 0) {
          atomicAdd(P.lost, 1ull);
          P.scores[C.pi] = 0; P.status[C.pi] = WFG_ST_DEVICE_ERROR; P.run_off[C.pi] = 0; P.run_len[C.pi] = 0;
          atomicSub(&B.active, 1);
        }
        return false;
      }
      __threadfence_block();
      __syncwarp();
      if (lane < 10) C.part[lane] = *(volatile int*)&S.job.part[lane];
      __syncwarp();
      C.d = S.job.d; C.t0 = S.job.t0;
      state = C.after;
      // the directions' rows
      const bool both = state == kSearch;
      if (lane < 4) {
        S.dir[C.d].ts.akr[((C.t0 >> 2) % 3) * 4 + lane] = max(C.part[lane], 0);
        if (both) R.ts.akr[((C.t0 >> 2) % 3) * 4 + lane] = max(C.part[5 + lane], 0);
      }
      tile_done(S.dir[C.d], C.t0, C.part[4]);
      if (both) tile_done(R, C.t0, C.part[9]);
      __syncwarp();
      if (state == kSearch) {
        // as behind the pass in the kernel: on to the next block unless a row may hold an event
        int nf = C.fmax, nr = C.rmax;
        #pragma unroll 1
        for (int j = 0; j < 4; ++j) { nf = max(nf, C.part[j]); nr = max(nr, C.part[5 + j]); }
        if (min(C.part[4], C.part[9]) == 4 && nf + nr < C.max_antidiag && C.t0 <= C.guard) {
          const int t0 = C.t0;
          if (tile_request<LIN>(0, true, t0 + 4, kSearch, gib, lane)) {
            C.fmax = nf; C.rmax = nr;
            __syncwarp();
            return true;
          }
        }
        state = kSearchEvent;
      }
    }
  }

  for (;;) {
    if (state == kFetch) {
      // The queue's head is dealt out block by block, so that a batch of few pairs spreads over all
      // thread blocks and each pair has helpers; the rest by one add per pair.
      int idx = -1;
      if (lane == 0 && gib < owners) {
        const unsigned long long n = P.num_pairs_ptr ? *P.num_pairs_ptr : (unsigned long long)P.num_pairs;
        unsigned long long w = (unsigned long long)gib * gridDim.x + blockIdx.x;
        if (!C.first) w = atomicAdd(P.queue_head, 1ull) + (unsigned long long)gridDim.x * owners;
        idx = w < n ? (int)w : -1;
      }
      idx = __shfl_sync(kFull, idx, 0);
      C.first = false;
      if (idx < 0) {
        if (lane == 0) { atomicSub(&B.active, 1); atomicAdd(&B.idle, 1); }
        C.state = state = kHelp;
        __syncwarp();
        continue;
      }
      const TileArena& A = S.arena;
      const int pi = P.order[idx];
      const PairDesc pd = P.pairs[pi];
      C.pi = pi;
      C.q.pf = P.words + pd.word_off;
      C.q.tf = C.q.pf + pd.pw_len;
      C.q.pr = C.q.tf + pd.tw_len;
      C.q.tr = C.q.pr + pd.pw_len;
      C.q.plen = pd.plen; C.q.tlen = pd.tlen; C.q.bshift = (pd.bits == 2) ? 1 : 3;
      // Rings sized to the pair: every wavefront of the pair (and of its sub-windows) lies on
      // diagonals [-plen-1, tlen+1]; the margin holds the last tile's unused lanes and the halos.
      const uint32_t need = (uint32_t)(pd.plen + pd.tlen + 8 + WFG_TILE_MARGIN);
      const int wp = min(P.ring_w, max(64, (int)(1u << (32 - __clz((int)need - 1)))));
      F.cfg.W = R.cfg.W = wp;
      F.cfg.pitch = R.cfg.pitch = wp + WFG_TILE_PAD;
      F.cfg.rdata = A.ring;
      R.cfg.rdata = A.ring + (size_t)P.ring_nphys * 3 * (wp + WFG_TILE_PAD);
      S.pen.tg = wp >= kTileMinRing ? P.tile_g : 0;
      C.status = ST_OK; C.score = 0;
      out.buf = A.runs; out.n = 0; out.cap = P.run_cap; out.cur_op = -1; out.cur_len = 0; out.overflow = false;
      C.pb = 0; C.pe = pd.plen; C.tb = 0; C.te = pd.tlen; C.cb = CM; C.ce = CM;
      C.rem = max(pd.plen, pd.tlen) <= kFallbackMinLength ? 0 : INT_MAX;  // short pairs take the leaf
      C.sp = 0;
      __syncwarp();
      state = P.score_only ? kSearch : kPop;
      if (state == kPop) {  // the root is the window at hand
        C.sp = -1;
        __syncwarp();
      }
    }

    if (state == kPop) {
      // wavefront_bialign_alignment's recursion on an explicit stack (half_0 before half_1)
      // sp is read once and written behind a barrier: a lane that still compares must not see the
      // root's -1 already replaced by 0, the empty stack.
      const int sp = C.sp;
      if (sp == 0 || C.status != ST_OK) {
        state = kFinish;
      } else {
        if (sp > 0) {
          const int4* e = reinterpret_cast<const int4*>(S.arena.stack + (sp - 1) * 8);
          const int4 a = e[0], b = e[1];
          __syncwarp();
          C.sp = sp - 1;
          C.pb = a.x; C.pe = a.y; C.tb = a.z; C.te = a.w;
          C.cb = b.x; C.ce = b.y; C.rem = b.z;
        } else {
          __syncwarp();
          C.sp = 0;
        }
        __syncwarp();
        const int pl = C.pe - C.pb, tl = C.te - C.tb;
        if (tl == 0) out.emit(WFG_OP_DEL, pl);
        else if (pl == 0) out.emit(WFG_OP_INS, tl);
        else state = C.rem <= kFallbackMinScore ? kLeaf : kSearch;
        if (state == kPop) continue;
      }
    }

    if (state == kSearch) {
      // wavefront_bialign_find_breakpoint: both directions' blocks until one may hold an event — the
      // antidiagonals add up, or a row touches an end
      C.guard = score_guard(pen, C.pe - C.pb, C.te - C.tb);
      C.max_antidiag = C.pe - C.pb + C.te - C.tb - 1;
      bp.score = INT_MAX;
      const SeqView fv = fwd_view(C.q, C.pb, C.pe, C.tb, C.te), rv = rev_view(C.q, C.pb, C.pe, C.tb, C.te);
      if (pen.tg == 0 || tile_start<LIN>(F, fv, C.cb, C.ce, lane) < 0 || tile_start<LIN>(R, rv, C.ce, C.cb, lane) < 0) {
        st = find_breakpoint<1, false>(F, R, C.q, C.pb, C.pe, C.tb, C.te, C.cb, C.ce, pen, P.max_steps, bp, g);
        state = kBpDone;
      } else {
        C.fmax = F.ts.akr[row_buffer(0)]; C.rmax = R.ts.akr[row_buffer(0)];
        C.sf = C.sr = 0;
        C.last_fwd = false;
        __syncwarp();
        if (C.fmax + C.rmax >= C.max_antidiag) {
          state = kMet;
        } else if (tile_request<LIN>(0, true, 0, kSearch, gib, lane)) {
          C.out = out; C.bp = bp;
          return true;
        } else {
          state = kSteps;
        }
      }
    }

    if (state == kSearchEvent) {
      // Replay of the block's rows up to the event; a touched row, or a full ring, leaves to the
      // single steps after the last row before it.
      if (!LIN && C.t0 >= kGapFirst) search_gaps(gib, lane);
      int t = C.t0, fmax = C.fmax, rmax = C.rmax, sf = 0, sr = 0;
      const int ft = C.part[4], rt = C.part[9];
      bool steps = true, last_fwd = false;
      #pragma unroll 1
      for (int j = 0; j < 4; ++j, ++t) {
        sf = sr = (t + 1) * pen.tg;
        if (ft == j) break;
        const int f1 = max(fmax, C.part[j]);
        if (f1 + rmax >= C.max_antidiag) { sr = sf - 1; last_fwd = true; steps = false; break; }
        if (rt == j) break;
        const int r1 = max(rmax, C.part[5 + j]);
        if (f1 + r1 >= C.max_antidiag) { steps = false; break; }
        fmax = f1; rmax = r1;
      }
      if (steps) sf = sr = t * pen.tg;
      __syncwarp();
      C.fmax = fmax; C.rmax = rmax; C.sf = sf; C.sr = sr; C.last_fwd = last_fwd;
      __syncwarp();
      state = steps ? kSteps : kMet;
    }

    if (state == kMeet) { state = kMet; resumed = true; }  // a block of the second phase has come in
    if (state == kMet) {
      // Second phase: the row stepped last (F's if last_fwd) against the other direction's, then
      // a step of the other.
      const int scope = pen.scope;
      int sf = C.sf, sr = C.sr;
      bool last_fwd = C.last_fwd;
      for (;;) {
        const int s0 = last_fwd ? sf : sr, s1 = last_fwd ? sr : sf;
        Dir& b = last_fwd ? R : F;
        if (!resumed) {
          if (s0 + max(s1 - (scope - 1), 0) - pen.go >= bp.score) { st = ST_OK; state = kBpDone; break; }
          if (holds_row(s0, pen)) tile_overlap<LIN>(last_fwd ? F : R, b, s0, s1, last_fwd, bp, pen, lane);
        }
        resumed = false;
        if (holds_row(s1 + 1, pen)) {
          const int t = row_of(s1 + 1, pen);
          if (t > b.ts.valid && !b.ts.touched && tile_request<LIN>(last_fwd ? 1 : 0, false, b.ts.t, kMeet, gib, lane)) {
            C.sf = sf; C.sr = sr; C.last_fwd = last_fwd;
            C.out = out; C.bp = bp;
            __syncwarp();
            return true;
          }
          if (t > b.ts.valid || (b.ts.touched && t == b.ts.valid)) { resume = last_fwd ? 1 : 2; state = kSteps; break; }
        }
        if (last_fwd) ++sr; else ++sf;
        last_fwd = !last_fwd;
        if (max(sf, sr) > C.guard + 2 * scope) { st = WFG_ST_UNATTAINABLE; state = kBpDone; break; }
      }
      __syncwarp();
      C.sf = sf; C.sr = sr; C.last_fwd = last_fwd;
      __syncwarp();
    }

    if (state == kSteps) {
      tile_describe<LIN>(F, C.sf, C.sf - pen.scope + 1, pen);
      tile_describe<LIN>(R, C.sr, C.sr - pen.scope + 1, pen);
      st = breakpoint_steps<1, false, LIN ? 2 : 1>(F, R, C.sf, C.sr, C.fmax, C.rmax, C.last_fwd, resume, C.guard, pen, P.max_steps,
                                            bp, g);
      resume = 0;
      state = kBpDone;
    }

    if (state == kBpDone) {
      __syncwarp();
      if (P.score_only) {
        // wavefront_bialign_compute_score (wavefront/wavefront_bialign.c:662-699)
        if (st == ST_OK || st == ST_END_REACHED) {
          const int wf = (st == ST_END_REACHED) ? (F.status == ST_END_REACHED ? F.status_score : R.status_score) : bp.score;
          C.score = classic_score(P.metric, P.match_o, C.q.plen, C.q.tlen, wf);
          C.status = WFG_ST_COMPLETED;
        } else {
          C.status = st;
        }
        state = kFinish;
      } else if (st == ST_OK) {
        const int bh = bp.of, bv = bp.of - bp.kf;
        const int sp = C.sp;
        if (sp + 2 > P.stack_cap) {
          C.status = WFG_ST_SCRATCH_OVERFLOW;
        } else {
          int4* e = reinterpret_cast<int4*>(S.arena.stack + sp * 8);
          e[0] = make_int4(C.pb + bv, C.pe, C.tb + bh, C.te);
          e[1] = make_int4(bp.comp, C.ce, bp.sr, 0);
          e[2] = make_int4(C.pb, C.pb + bv, C.tb, C.tb + bh);
          e[3] = make_int4(C.cb, bp.comp, bp.sf, 0);
          __syncwarp();
          C.sp = sp + 2;
        }
        state = kPop;
      } else if (st == ST_END_REACHED) {
        const int reached = (F.status == ST_END_REACHED) ? F.status_score : R.status_score;
        state = reached <= kRecoveryMinScore ? kLeaf : kPop;
        if (state == kPop) C.status = WFG_ST_UNATTAINABLE;
      } else {
        C.status = (st == WFG_ST_SCRATCH_OVERFLOW || st == WFG_ST_MAX_STEPS || st == WFG_ST_OOM) ? st : WFG_ST_UNATTAINABLE;
        state = kPop;
      }
      __syncwarp();
      if (state == kPop) continue;
    }

    if (state == kLeaf) {
      // The leaf's rows in tiles, up to its end or the first touched row that is not its end; the
      // ring of F holds the rows that the next block reads, the leaf store gets every row.
      const SeqView sv = fwd_view(C.q, C.pb, C.pe, C.tb, C.te);
      C.guard = score_guard(pen, C.pe - C.pb, C.te - C.tb);
      const int off0 = pen.tg ? tile_start<LIN>(F, sv, C.cb, C.ce, lane) : -1;
      if (off0 < 0) {
        st = leaf_align<1, false>(L, C.q, C.pb, C.pe, C.tb, C.te, C.cb, C.ce, pen, P.max_steps, out,
                                  S.arena.lruns, P.leaf_run_cap, g, &s);
        __syncwarp();
        if (st != ST_OK) C.status = st;
        __syncwarp();
        state = kPop;
        continue;
      }
      if (lane == 0) L.cfg.ldata[0] = off0;
      L.sv = sv; L.cb = C.cb; L.ce = C.ce; L.num_null = 0; L.status = ST_OK; L.end_k = sv.tlen - sv.plen;
      C.leaf_end = leaf_at<LIN>(0, pen);
      __syncwarp();
      state = kLeafSteps;
      s = 0; done = false;
      if (4 * pen.tg <= L.cfg.lmax && leaf_at<LIN>(1, pen) <= L.lcap && tile_request<LIN>(0, false, 0, kLeaf, gib, lane)) {
        C.out = out; C.bp = bp;
        __syncwarp();
        return true;
      }
    }

    if (state == kLeafEvent) {
      // a touched row, or no room for another block
      const int t0 = C.t0, touch = C.part[4], last = touch < 4 ? t0 + 1 + touch : t0 + 4, ci = comp_index(C.ce);
      const int ak = L.end_k;
      s = last * pen.tg;
      if (touch < 4 && row_exists<LIN>(C.cb, last, ci, pen) && row_lo<LIN>(C.cb, last, pen) <= ak &&
          ak <= row_hi<LIN>(C.cb, last, pen))
        done = L.cfg.ldata[leaf_cell<LIN>(C.cb, last, ci, ak, pen)] >= L.sv.tlen;
      state = kLeafSteps;
    }

    if (state == kLeafSteps) {
      const int fast = s;
      __syncwarp();
      L.lused = C.leaf_end;
      L.status = done ? ST_END_REACHED : ST_OK;
      __syncwarp();
      st = ST_OK;
      if (!done) {
        leaf_describe<LIN>(L, s, s - pen.scope + 1, pen, lane);
        st = leaf_steps<1, false>(L, &s, C.guard, pen, P.max_steps, g);
      }
      if (st == ST_OK) st = tile_backtrace<LIN>(L, pen, s, fast, out, S.arena.lruns, P.leaf_run_cap, lane);
      __syncwarp();
      if (st != ST_OK) C.status = st;
      __syncwarp();
      done = false;
      state = kPop;
      continue;
    }

    if (state == kFinish) {
      int status = C.status, score = P.score_only ? C.score : 0;
      const int pi = C.pi;
      if (!P.score_only) {
        out.flush();
        if (status == ST_OK && out.overflow) status = WFG_ST_SCRATCH_OVERFLOW;
        if (status == ST_OK) status = WFG_ST_COMPLETED;
        __syncwarp();
        if (status == WFG_ST_COMPLETED) {
          // cigar_score_gap_affine (alignment/cigar.c:277-303) over maximal runs, a lane's runs each
          if (LIN && out.n > 0)
            score = rescore_runs(out.buf, out.n, P.metric, P.match_o, P.x_o, P.o_o, P.e_o, P.o2_o, P.e2_o);
          #pragma unroll 1
          for (int i = lane; !LIN && i < out.n; i += 32) {
            const int op = (int)(out.buf[i] & 15u), len = (int)(out.buf[i] >> 4);
            score -= op == WFG_OP_EQ ? P.match_o * len : op == WFG_OP_X ? P.x_o * len : P.o_o + P.e_o * len;
          }
          if (!LIN) score = __reduce_add_sync(kFull, score);
          unsigned long long base = 0;
          if (lane == 0) base = atomicAdd(P.out_head, (unsigned long long)out.n);
          base = __shfl_sync(kFull, base, 0);
          if ((long long)base + out.n > P.out_cap) {
            status = WFG_ST_OUTPUT_OVERFLOW;
          } else {
            #pragma unroll 1
            for (int i = lane; i < out.n; i += 32) P.out_runs[base + i] = out.buf[i];
            if (lane == 0) { P.run_off[pi] = (int64_t)base; P.run_len[pi] = out.n; }
          }
        }
      }
      if (status == WFG_ST_SCRATCH_OVERFLOW && P.retry_out != nullptr) {
        // Hand the pair to the next pass (larger arena); its results are written there.
        if (lane == 0) P.retry_out[atomicAdd(P.retry_count, 1ull)] = pi;
      } else if (lane == 0) {
        P.scores[pi] = score;
        P.status[pi] = status;
        if (status != WFG_ST_COMPLETED || P.score_only) { P.run_off[pi] = 0; P.run_len[pi] = 0; }
      }
      __syncwarp();
      state = kFetch;
      continue;
    }

    if (state == kHelp) {
      // Queue empty: tiles of the block's other warps until none has a pair.
      for (int spins = 0; spins < kSpinLimit && warp_read(B.active, lane) > 0; ++spins) {
        #pragma unroll 1
        for (int k = 1; k < kTileWarps; ++k) {
          const int w = gib + k < kTileWarps ? gib + k : gib + k - kTileWarps;
          const int i = job_take(B.grp[w].job, lane);
          if (i >= 0) { job_block(w, i, C); __syncwarp(); return true; }
        }
        __nanosleep(200);
      }
      if (lane == 0) atomicSub(&B.idle, 1);
      return false;
    }
  }
}

}  // namespace

// LIN: the one-component distances (edit, indel, gap-linear); else gap-affine.
template <bool LIN>
__global__ void __launch_bounds__(kTileWarps * 32, kTileBlocks) biwfa_tile_kernel(KernelParams Pin) {
  TileBlockSmem& B = tile_smem();
  if (Pin.num_pairs_ptr != nullptr && *Pin.num_pairs_ptr == 0ull) return;  // a retry pass without pairs
  const int gib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int owners = Pin.tile_owners;
  TileGroup& S = B.grp[gib];
  TileCtl& C = S.ctl;
  if (threadIdx.x == 0) { B.P = Pin; B.active = owners; B.idle = kTileWarps - owners; }
  {
    const ArenaLayout L = wfg_arena_layout(Pin.ring_nphys, Pin.ring_w + WFG_TILE_PAD, Pin.leaf_max_score, Pin.leaf_words,
                                           Pin.run_cap, Pin.leaf_run_cap, Pin.stack_cap, 3);
    uint8_t* arena = Pin.arena + ((long long)blockIdx.x * owners + min(gib, owners - 1)) * Pin.arena_bytes;
    TileArena A;
    A.ring = (int32_t*)(arena + L.ring_off);
    A.ldesc = (int4*)(arena + L.ldesc_off); A.ldata = (int32_t*)(arena + L.ldata_off);
    A.runs = (uint32_t*)(arena + L.runs_off); A.lruns = (uint32_t*)(arena + L.lruns_off);
    A.stack = (int*)(arena + L.stack_off);
    DirCfg c{};
    c.scope = Pin.scope; c.magic = (uint32_t)(0xffffffffu / (uint32_t)Pin.scope) + 1u;
    c.nphys = Pin.ring_nphys; c.nc = 3;
    if (lane < 2) {
      c.rdesc = S.rdesc[lane]; c.rphys = S.rphys[lane];
    } else {
      c.leaf = 1; c.nphys = 1; c.lmax = Pin.leaf_max_score; c.ldesc = A.ldesc; c.ldata = A.ldata;
    }
    if (lane < 3) {
      Dir& d = S.dir[lane];
      d.cfg = c;
      d.lused = 0; d.lcap = lane == 2 ? Pin.leaf_words : 0;
      d.ts.on = 0;
    }
    if (lane == 0) {
      S.arena = A;
      S.pen = {Pin.x, Pin.o, Pin.e, Pin.scope, Pin.metric, LIN ? 0 : Pin.o, 0,
               Pin.tile_g > 1 ? 0xffffffffu / (uint32_t)Pin.tile_g + 1u : 0u};
      if (LIN) {
        S.pen.lx = Pin.metric == kMetricIndel ? 0 : Pin.x / Pin.tile_g;
        S.pen.lo = Pin.o / Pin.tile_g;
        S.pen.lom = 0xffffffffu / (uint32_t)S.pen.lo + 1u;
      }
      S.job.ticket = 0ull;
      C.state = gib < owners ? kFetch : kHelp;
      C.first = true;
      C.step = 0;
      C.owner = gib;
    }
  }
  __syncthreads();

  bool control = true;
  for (;;) {
    if (control && !tile_control<LIN>(gib, lane, owners)) break;
    control = true;
    if (C.step == 0) continue;  // an own job whose tiles the helpers took
    // ---- the block pass
    const int mode = C.mode, t0 = C.t0, d0 = C.d;
    const bool halves = mode == kHalves, upper = lane >= 16;
    const int L = halves ? 16 : 32, tl = lane & (L - 1), b = (t0 >> 2) % 3;
    const bool leaf = C.state == kLeaf;
    int part[2], touch[2];  // lanes 0-3: largest antidiagonal of each row; first touched row
    part[1] = INT_MIN; touch[1] = 4;
    #pragma unroll 1
    for (int x = 0; x < (mode == kBoth ? 2 : 1); ++x) {
      const Dir& my = B.grp[C.owner].dir[(halves && upper) || x ? 1 : d0];
      const SeqView sv = my.sv;
      const int tiles = my.ts.tiles, narrow = my.ts.narrow;
      TileArgs a;
      a.pitch = my.cfg.pitch;
      a.old_rows = my.cfg.rdata + wfg_tile_row((b == 0 ? 2 : b - 1) * 12, a.pitch);
      a.new_rows = my.cfg.rdata + wfg_tile_row(b * 12, a.pitch);
      a.mask = (uint32_t)my.cfg.W - 1u;
      a.old_lo = my.ts.lo; a.old_hi = my.ts.hi;
      a.first = tl == 0; a.last = tl == L - 1;
      a.lane = lane;
      a.gaps = my.ts.gaps;
      if (LIN) { a.lx = S.pen.lx; a.lo = S.pen.lo; }
      a.leaf = leaf ? S.dir[2].cfg.ldata + leaf_at<LIN>(t0 >> 2, S.pen) : nullptr;
      a.leaf_lo = leaf_lo<LIN>(my.cb, t0 >> 2, S.pen); a.leaf_n = leaf ? leaf_n<LIN>(t0 >> 2, S.pen) : 0;
      int ak = INT_MIN, tch = 4;
      const int step = C.step;
      int i = C.tile;
      a.k = my.ts.base + tl * 4;
      a.owner = tiles == 1 || !(a.first || a.last);
      #pragma unroll 1
      for (; i < tiles - narrow; i += step)
        tile_pass<4, LIN>(a, sv, i * 120, a.owner || (i == 0 && a.first) || (i == tiles - 1 && a.last), ak, tch);
      if (i < tiles) {  // the last tile, two diagonals per lane
        a.k = my.ts.base + tl * 2;
        a.owner = tiles == 1 || (tl >= 2 && tl < L - 2);
        tile_pass<2, LIN>(a, sv, i * 120, a.owner || tl >= L - 2 || i == 0, ak, tch);
      }
      const int other = __shfl_xor_sync(kFull, ak, 16);
      if (halves) {
        part[0] = ak; part[1] = other;
        touch[0] = __reduce_min_sync(kFull, upper ? 4 : tch);
        touch[1] = __reduce_min_sync(kFull, upper ? tch : 4);
      } else {
        part[x] = max(ak, other);
        touch[x] = __reduce_min_sync(kFull, tch);
      }
    }
    if (lane < 4) { C.part[lane] = part[0]; C.part[5 + lane] = part[1]; }
    if (lane == 4) { C.part[4] = touch[0]; C.part[9] = touch[1]; }
    const int state = C.state;
    if (state == kHelp || state == kOwnJob) {  // the tile goes to its job; on to the next one
      __syncwarp();
      TileJob& job = B.grp[C.owner].job;
      job_add(C, lane);
      const int i = job_take(job, lane);
      if (i >= 0) job_block(C.owner, i, C);
      else C.step = 0;
      control = i < 0;
      __syncwarp();
      continue;
    }
    // ---- the rows' state, and the common continuations
    const bool both = mode != kOne;
    if (lane < 4) {
      S.dir[d0].ts.akr[b * 4 + lane] = max(part[0], 0);
      if (both) S.dir[1].ts.akr[b * 4 + lane] = max(part[1], 0);
    }
    tile_done(S.dir[d0], t0, touch[0]);
    if (both) tile_done(S.dir[1], t0, touch[1]);
    __syncwarp();
    if (state == kSearch) {
      const int nf = max(C.fmax, __reduce_max_sync(kFull, lane < 4 ? part[0] : INT_MIN));
      const int nr = max(C.rmax, __reduce_max_sync(kFull, lane < 4 ? part[1] : INT_MIN));
      if (min(touch[0], touch[1]) == 4 && nf + nr < C.max_antidiag && t0 <= C.guard &&
          tile_request<LIN>(0, true, t0 + 4, kSearch, gib, lane)) {
        C.fmax = nf; C.rmax = nr;
        control = false;
      } else {
        C.state = kSearchEvent;
      }
    } else if (state == kLeaf) {
      const int end = leaf_at<LIN>((t0 >> 2) + 1, S.pen);
      C.leaf_end = end;
      if (touch[0] == 4 && t0 <= C.guard && (t0 + 8) * S.pen.tg <= S.dir[2].cfg.lmax &&
          leaf_at<LIN>((t0 >> 2) + 2, S.pen) <= S.dir[2].lcap && tile_request<LIN>(0, false, t0 + 4, kLeaf, gib, lane)) {
        control = false;
      } else {
        C.state = kLeafEvent;
      }
    }
    __syncwarp();
  }
}
