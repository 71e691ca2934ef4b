// Wavefront rows in tiles: four score steps of a direction per pass over its diagonals.
// Included by biwfa_kernel.cu inside its anonymous namespace.
//
// Every score that can hold a wavefront is a multiple of g = gcd(x, o+e, e); a row is t = s / g.
// For penalties with x = 2g, o+e = 4g, e = g (4/6/2, the defaults, and 2/3/1) row t needs M of
// rows t-2 and t-4 and I, D of row t-1, so a lane that holds M of the last four rows and I, D of
// the last one in registers computes the next four rows with one shuffle per component and row:
// the rows are read and written once per four steps, in 16-byte vectors, and everything that a
// step pays once (descriptors, reductions, calls) is paid once per four.
//
//   tile   L lanes x C adjacent diagonals: half a warp per direction (both directions in one
//          pass) while their wavefronts are narrow, else a warp; a wavefront of several tiles
//          gives each a halo of four diagonals per side, recomputed by the neighbour tile
//   block  rows t0+1 .. t0+4 of one direction (t0 a multiple of 4)
//   ring   kTileBufs = 12 physical buffers, row t in buffer (t - 1) mod 12: a block reads one
//          group of four buffers and writes the next; the diagonals that the last block wrote are
//          known, all others are null
//
// What bounds it: instruction issue and fetch, then the latency of a row's two dependent rounds
// (shuffles, then the sequence windows). One score at a time cost about 264 lane instructions per
// diagonal and row, 40 % of them paid per step; a tile costs about 60. End to end on a GB300, one
// score at a time -> tiles: 10,000 pairs of 1 kbp at 5 % 7.7 -> 3.8 ms, 20,000 uneven pairs
// (100 bp - 10 kbp, 1-10 %) 320 -> 102 ms, 48 pairs of 10-20 kbp at 12 % (8 warps per pair)
// 569 -> 135 ms, 200,000 pairs of 150 bp at 2 % 15.3 -> 13.4 ms.
//
// Where the values are exact. WFA2-lib trims each row to its in-bounds cells and keeps
// out-of-bounds I/D cells between them. Out-of-bounds cells arise only from a cell whose offset
// has reached the end of the pattern or of the text ("touches": no further extension possible).
// So up to and including the first touched row all values are in bounds or null, trimming only
// removes nulls, and the rows here equal WFA2-lib's with its nulls (any negative offset is null).
// From the row after it the one-step functions (dir_step) continue from the stored rows.

constexpr int kTNull = -(1 << 28);  // null offset of a row; the few units it drifts never make it positive
constexpr int kTileHalo = 4;
constexpr int kTX = 2, kTO = 4;     // rows back to the mismatch and the gap-opening source
constexpr int kTileMinRing = 256;   // narrowest ring that is worth tiles

// Row of score s (rounded down) and whether s has one. The spacing is at most 8 and scores stay
// below 2^27, so the product with tm = floor(2^32 / tg) + 1 divides exactly.
__device__ __forceinline__ int row_of(int s, const Pen& p) { return p.tg == 1 ? s : (int)__umulhi((uint32_t)s, p.tm); }
__device__ __forceinline__ bool holds_row(int s, const Pen& p) { return s == row_of(s, p) * p.tg; }

// Diagonals that can hold a non-null cell in row t of a direction that starts in component cb
// (the rows of all components lie inside; both bounds widen monotonically).
__device__ __forceinline__ int row_lo(int cb, int t) {
  return cb == CM ? (t < kTO ? 0 : kTO - 1 - t) : cb == CI ? min(0, kTO + 1 - t) : -t;
}
__device__ __forceinline__ int row_hi(int cb, int t) {
  return cb == CM ? (t < kTO ? 0 : t - kTO + 1) : cb == CI ? t : max(0, t - kTO - 1);
}
// Whether component ci (0 M, 1 I, 2 D) of row t exists: some cell of it is not null.
__device__ __forceinline__ bool row_exists(int cb, int t, int ci) {
  if (t < 0) return false;
  if (cb == CM) return ci == 0 ? (t >= kTO || t % kTX == 0) : t >= kTO;
  if (ci == 0) return t >= 1;
  return ci == (cb == CI ? 1 : 2) ? true : t >= kTO + 1;
}
__device__ __forceinline__ int row_buffer(int t) { return (t + kTileBufs - 1) % kTileBufs; }

template <int C> struct TileVec;
template <> struct TileVec<1> { typedef int type; };
template <> struct TileVec<2> { typedef int2 type; };
template <> struct TileVec<4> { typedef int4 type; };
template <int C>
__device__ __forceinline__ void tile_load(const int32_t* p, int (&v)[C]) {
  if (C == 1) { v[0] = *p; }
  else if (C == 2) { const int2 q = *reinterpret_cast<const int2*>(p); v[0] = q.x; v[C - 1] = q.y; }
  else { const int4 q = *reinterpret_cast<const int4*>(p); v[0] = q.x; v[1 % C] = q.y; v[2 % C] = q.z; v[3 % C] = q.w; }
}
template <int C>
__device__ __forceinline__ void tile_store(int32_t* p, const int (&v)[C]) {
  if (C == 1) *p = v[0];
  else if (C == 2) *reinterpret_cast<int2*>(p) = make_int2(v[0], v[C - 1]);
  else *reinterpret_cast<int4*>(p) = make_int4(v[0], v[1 % C], v[2 % C], v[3 % C]);
}

// What a pass over one block's tiles needs. A lane's own direction: in a pass over both
// directions the lower half warp holds F's diagonals and the upper half R's.
struct TileArgs {
  int32_t* old_rows;   // buffer group of rows t0-3 .. t0
  int32_t* new_rows;   // buffer group of rows t0+1 .. t0+4
  int32_t* leaf;       // leaf store of rows t0+1 .. t0+4 (M, I, D each), diagonals [leaf_lo, leaf_lo + leaf_n)
  int leaf_lo, leaf_n; // leaf_n 0: no leaf store
  int pitch;
  uint32_t mask;
  int old_lo, old_hi;  // diagonals that the old rows hold (multiples of 4)
  int k;               // this lane's first diagonal in the first tile
  bool first, last;    // this lane is the first or last one of its tile
  bool owner;          // this lane's diagonals are not halo
  int lane;
};

// Rows t0+1 .. t0+4 of a tile's diagonals, a.k + off in this lane. Lanes j and 16 + j of ak: the
// largest antidiagonal of row t0+1+j in the lower and the upper half warp; touch: the first of the
// four rows (0-3) where this lane touched, else unchanged. The loop over the rows stays rolled (the
// last four rows' registers rotate by moves): unrolled, the warps' instructions did not fit the
// instruction caches, and waiting for them took 76 % of the issue slots.
template <int C>
__device__ __forceinline__ void tile_pass(const TileArgs& a, const SeqView& sv, int off, bool store, int& ak, int& touch) {
  const int k0 = a.k + off;
  const uint32_t idx = (uint32_t)k0 & a.mask;
  const int p3 = 3 * a.pitch;
  int m[4][C], vi[C], vd[C];
  if (k0 >= a.old_lo && k0 < a.old_hi) {
    #pragma unroll
    for (int j = 0; j < 4; ++j) tile_load<C>(a.old_rows + j * p3 + idx, m[j]);
    tile_load<C>(a.old_rows + 3 * p3 + a.pitch + idx, vi);
    tile_load<C>(a.old_rows + 3 * p3 + 2 * a.pitch + idx, vd);
  } else {
    #pragma unroll
    for (int c = 0; c < C; ++c) m[0][c] = m[1][c] = m[2][c] = m[3][c] = vi[c] = vd[c] = kTNull;
  }
  const int wsh = 5 - sv.bshift, cpw = 32 >> sv.bshift;
  const bool leafw = a.owner && (unsigned)(k0 - a.leaf_lo) < (unsigned)a.leaf_n;
  int32_t* ring = a.new_rows + idx;
  int32_t* leaf = a.leaf + (k0 - a.leaf_lo);
  #pragma unroll 1
  for (int j = 0; j < 4; ++j) {
    // I = max(M[t-4], I[t-1])[k-1] + 1, D = max(M[t-4], D[t-1])[k+1], M = max(M[t-2] + 1, I, D)
    int fi[C], fd[C], n[C];
    uint32_t x[C];
    #pragma unroll
    for (int c = 0; c < C; ++c) { fi[c] = max(m[4 - kTO][c], vi[c]); fd[c] = max(m[4 - kTO][c], vd[c]); }
    int left = __shfl_up_sync(kFull, fi[C - 1], 1), right = __shfl_down_sync(kFull, fd[0], 1);
    if (a.first) left = kTNull;
    if (a.last) right = kTNull;
    #pragma unroll
    for (int c = 0; c < C; ++c) {
      vi[c] = (c == 0 ? left : fi[c > 0 ? c - 1 : 0]) + 1;
      vd[c] = (c == C - 1 ? right : fd[c < C - 1 ? c + 1 : C - 1]);
      n[c] = max(m[4 - kTX][c] + 1, max(vi[c], vd[c]));
    }
    // First windows of all cells (a null cell reads the sequences' starts).
    #pragma unroll
    for (int c = 0; c < C; ++c) {
      const int pp = max(n[c] + (sv.p0 - k0 - c), sv.p0), tt = max(n[c] + sv.t0, sv.t0);
      const uint32_t wp = (uint32_t)pp >> wsh, wt = (uint32_t)tt >> wsh;
      x[c] = __funnelshift_r(seq_word(sv.pw, wp), seq_word(sv.pw, wp + 1), (uint32_t)pp << sv.bshift) ^
             __funnelshift_r(seq_word(sv.tw, wt), seq_word(sv.tw, wt + 1), (uint32_t)tt << sv.bshift);
    }
    uint32_t more = 0;
    bool ends = false;
    #pragma unroll
    for (int c = 0; c < C; ++c) {
      const int rem = min(sv.tlen, sv.plen + k0 + c) - n[c];  // to the end of diagonal k0 + c
      int e = x[c] ? (first_set(x[c]) >> sv.bshift) : cpw;
      if (x[c] == 0 && rem > cpw && n[c] >= 0) more |= 1u << c;
      e = min(e, rem);
      ends |= e >= rem;
      n[c] += e;
    }
    // Matches longer than one window.
    #pragma unroll 1
    while (more) {
      const int c = __ffs((int)more) - 1;
      more &= more - 1;
      int cur = n[0];
      #pragma unroll
      for (int i = 1; i < C; ++i) if (c == i) cur = n[i];
      const int dk = sv.p0 - k0 - c, end = min(sv.tlen, sv.plen + k0 + c);
      #pragma unroll 1
      while (cur < end) {
        const int pp = cur + dk, tt = cur + sv.t0;
        const uint32_t wp = (uint32_t)pp >> wsh, wt = (uint32_t)tt >> wsh;
        const uint32_t y = __funnelshift_r(seq_word(sv.pw, wp), seq_word(sv.pw, wp + 1), (uint32_t)pp << sv.bshift) ^
                           __funnelshift_r(seq_word(sv.tw, wt), seq_word(sv.tw, wt + 1), (uint32_t)tt << sv.bshift);
        if (y) { cur += first_set(y) >> sv.bshift; break; }
        cur += cpw;
      }
      cur = min(cur, end);
      ends |= cur >= end;
      #pragma unroll
      for (int i = 0; i < C; ++i) if (c == i) n[i] = cur;
    }
    if (ends) touch = min(touch, j);
    int best = 2 * n[0];
    #pragma unroll
    for (int c = 1; c < C; ++c) best = max(best, 2 * n[c] - c);
    best -= k0;
    const int lower = __reduce_max_sync(kFull, a.lane < 16 ? best : INT_MIN);
    const int upper = __reduce_max_sync(kFull, a.lane < 16 ? INT_MIN : best);
    if ((a.lane & 15) == j) ak = max(ak, a.lane < 16 ? lower : upper);
    #pragma unroll
    for (int c = 0; c < C; ++c) { m[0][c] = m[1][c]; m[1][c] = m[2][c]; m[2][c] = m[3][c]; m[3][c] = n[c]; }
    if (store) {
      tile_store<C>(ring, n);
      if (a.leaf_n == 0 || j == 3) { tile_store<C>(ring + a.pitch, vi); tile_store<C>(ring + 2 * a.pitch, vd); }
    }
    ring += p3;
    if (leafw) {
      tile_store<C>(leaf, n);
      tile_store<C>(leaf + a.leaf_n, vi);
      tile_store<C>(leaf + 2 * a.leaf_n, vd);
    }
    leaf += 3 * a.leaf_n;
  }
}

// The tiling of one block for L lanes: tiles, first diagonal, end of the last tile. One tile of
// 4 L diagonals if they hold all of the rows' cells (the cells beside it are null), else tiles with
// halos.
struct TilePlan { int tiles, base, end; };
__device__ __forceinline__ TilePlan tile_plan(int cb, int t0, int L) {
  TilePlan p;
  const int lo = row_lo(cb, t0 + 4) & ~3, width = row_hi(cb, t0 + 4) - lo + 1;
  p.tiles = 1; p.base = lo;
  if (width > 4 * L) { p.tiles = (width + 119) / 120; p.base = lo - kTileHalo; }
  p.end = p.base + (p.tiles - 1) * 120 + 4 * L;
  return p;
}

// One warp's tiles (first, first + step, ...) of block t0 of direction d, or (pair) the tile of
// both d and e, narrow enough for half a warp each. The warp's largest antidiagonal of each row and
// first touched row (4: none) go to part[0..4]; with pair, e's to part_e.
__device__ __noinline__ void tile_run(const Dir& d, const Dir& e, bool pair, int t0, int first, int step, int32_t* leaf,
                                      int leaf_lo, int leaf_n, int lane, int* part, int* part_e) {
  const bool upper = lane >= 16;
  const Dir& my = pair && upper ? e : d;
  const int L = pair ? 16 : 32, tl = lane & (L - 1);
  const TilePlan p = tile_plan(my.cb, t0, L);
  const SeqView sv = my.sv;
  TileArgs a;
  const int b = (t0 >> 2) % 3;
  a.pitch = my.cfg.pitch;
  a.old_rows = my.cfg.rdata + (b == 0 ? 2 : b - 1) * 12 * a.pitch;
  a.new_rows = my.cfg.rdata + b * 12 * a.pitch;
  a.mask = (uint32_t)my.cfg.W - 1u;
  a.old_lo = my.ts.lo; a.old_hi = my.ts.hi;
  a.first = tl == 0; a.last = tl == L - 1;
  a.lane = lane;
  a.leaf = leaf; a.leaf_lo = leaf_lo; a.leaf_n = leaf_n;
  int ak = INT_MIN, touch = 4;
  // two diagonals per lane while they hold the rows (in both directions of a pair)
  const bool narrow = row_hi(my.cb, t0 + 4) - p.base < 2 * L && p.tiles == 1;
  if (__all_sync(kFull, narrow)) {
    a.k = p.base + tl * 2;
    a.owner = true;
    if (first == 0) tile_pass<2>(a, sv, 0, true, ak, touch);
  } else {
    a.k = p.base + tl * 4;
    a.owner = p.tiles == 1 || !(a.first || a.last);
    #pragma unroll 1
    for (int i = first; i < p.tiles; i += step)
      tile_pass<4>(a, sv, i * 120, a.owner || (i == 0 && a.first) || (i == p.tiles - 1 && a.last), ak, touch);
  }
  const int t_lo = __reduce_min_sync(kFull, upper ? 4 : touch), t_up = __reduce_min_sync(kFull, upper ? touch : 4);
  const int other = __shfl_xor_sync(kFull, ak, 16);
  if (pair) {
    int* out = upper ? part_e : part;
    if ((lane & 15) < 4) out[lane & 15] = ak;
    if ((lane & 15) == 4) out[4] = upper ? t_up : t_lo;
  } else {
    if (lane < 4) part[lane] = max(ak, other);
    if (lane == 4) part[4] = min(t_lo, t_up);
  }
}

// The diagonals that block t0 writes (tile_run's choice of tiles).
__device__ __forceinline__ void tile_span(int cb, int t0, bool pair, bool narrow, int& lo, int& hi) {
  const TilePlan p = tile_plan(cb, t0, pair ? 16 : 32);
  lo = p.base;
  hi = narrow ? p.base + (pair ? 32 : 64) : p.end;
}
__device__ __forceinline__ bool tile_narrow(int cb, int t0, int L) {
  return row_hi(cb, t0 + 4) - (row_lo(cb, t0 + 4) & ~3) < 2 * L;
}
// Whether the ring holds block t0's diagonals.
__device__ __forceinline__ bool tile_fits(const Dir& d, int t0) {
  const TilePlan p = tile_plan(d.cb, t0, 32);
  return p.end - p.base <= d.cfg.W;
}

// The first extension of a direction's diagonal 0.
__device__ __noinline__ int first_match(const uint32_t* pw, const uint32_t* tw, int p0, int t0, int n, int bshift) {
  SeqView v;
  v.pw = pw; v.tw = tw; v.p0 = p0; v.t0 = t0; v.plen = n; v.tlen = n; v.bshift = bshift;
  return lcp(v, 0, 0);
}

// Starts a direction over window sv in component cb: row 0 with its extension. Returns its offset,
// or -1 when it touches (then nothing is started). The caller syncs before and after it.
template <int G>
__device__ __noinline__ int tile_start(Dir& d, const SeqView& sv, int cb, int ce, const Grp<G> g) {
  const int n = min(sv.plen, sv.tlen);
  const int off0 = cb == CM ? first_match(sv.pw, sv.tw, sv.p0, sv.t0, n, sv.bshift) : 0;
  if (off0 >= n) return -1;
  d.sv = sv; d.cb = cb; d.ce = ce;
  d.num_null = 0; d.status = ST_OK; d.status_score = 0; d.end_k = INT_MAX;
  d.ts.on = 1; d.ts.t = 0; d.ts.valid = 0; d.ts.touched = 0;
  d.ts.lo = 0; d.ts.hi = 4;
  d.ts.akr[row_buffer(0)] = cb == CM ? 2 * off0 : 0;
  // rows -3 .. 0 on diagonals 0-3: M in buffers 8-11, I and D of row 0
  if (g.tid < 6) {
    const int row = g.tid < 4 ? (8 + g.tid) * 3 : 11 * 3 + g.tid - 3;
    const int mine = g.tid < 3 ? -1 : g.tid - 3;  // the component of row 0
    *reinterpret_cast<int4*>(d.cfg.rdata + row * d.cfg.pitch) =
        make_int4(mine == comp_index(cb) ? off0 : kTNull, kTNull, kTNull, kTNull);
  }
  return off0;
}

// Combines the warps' parts of a block (after a group barrier): antidiagonals into the rows'
// entries; returns the first touched row of the four, 4 if none.
template <int G>
__device__ __forceinline__ int tile_combine(Dir& d, int t0, const int* part, const Grp<G>& g) {
  int touch = part[4];
  #pragma unroll
  for (int w = 1; w < G; ++w) touch = min(touch, part[w * 5 + 4]);
  if (g.lane() < 4) {
    int v = part[g.lane()];
    #pragma unroll
    for (int w = 1; w < G; ++w) v = max(v, part[w * 5 + g.lane()]);
    d.ts.akr[((t0 >> 2) % 3) * 4 + g.lane()] = max(v, 0);
  }
  __syncwarp();
  return touch;
}

// The state after block t0 (touch as tile_combine gives it). Callers pass a group barrier between
// the last read of d.ts and this.
__device__ __forceinline__ void tile_done(Dir& d, int t0, int touch, bool pair, bool narrow) {
  int lo, hi;
  tile_span(d.cb, t0, pair, narrow, lo, hi);
  d.ts.lo = lo; d.ts.hi = hi;
  d.ts.t = t0 + 4;
  d.ts.touched = touch < 4 ? 1 : 0;
  d.ts.valid = touch < 4 ? t0 + 1 + touch : t0 + 4;
}

// The next block of one direction; false when the ring is full.
template <int G>
__device__ __noinline__ bool tile_next(Dir& d, const Grp<G> g, int* part) {
  const int t0 = d.ts.t;
  if (!tile_fits(d, t0)) return false;
  int* mine = part + ((t0 >> 2) & 1) * (G * 5);
  tile_run(d, d, false, t0, g.warp(), G, nullptr, 0, 0, g.lane(), mine + g.warp() * 5, nullptr);
  g.sync();
  const int touch = tile_combine<G>(d, t0, mine, g);
  tile_done(d, t0, touch, false, tile_narrow(d.cb, t0, 32));
  return true;
}

// Descriptors of the scores from .. s from their rows (a score without a row is absent).
__device__ __noinline__ void tile_describe(Dir& d, int s, int from, const Pen& p) {
  const DirCfg c = d.cfg;
  #pragma unroll 1
  for (int q = max(from, 0); q <= s; ++q) {
    const int slot = slot_of(c, q), t = row_of(q, p);
    const bool row = holds_row(q, p);
    const int lo = row_lo(d.cb, t), hi = row_hi(d.cb, t);
    #pragma unroll 1
    for (int ci = 0; ci < 3; ++ci)
      c.rdesc[slot * 3 + ci] = row && row_exists(d.cb, t, ci) ? make_int2(lo, hi) : make_int2(kAbsent, INT_MIN);
    c.rphys[slot] = row_buffer(t);
  }
}

// Step of a direction to score s with its descriptors: from the rows computed ahead, from a new
// block, or — once the rows have touched or the ring is full — by dir_step. Returns as dir_step.
template <int G>
__device__ __noinline__ int tile_advance(Dir& d, const Pen p, int s, const Grp<G> g, int* part, int* max_ak_out) {
  *max_ak_out = 0;
  if (d.ts.on) {
    const bool row = holds_row(s, p);
    const int t = row_of(s, p);
    if (!row || t <= d.ts.valid || (!d.ts.touched && tile_next<G>(d, g, part))) {
      if (G > 1) g.sync();
      tile_describe(d, s, s, p);
      g.sync();
      if (!row) return 0;
      if (d.ts.touched && t == d.ts.valid) {
        const int ak = d.sv.tlen - d.sv.plen;
        const WfRef w = ref_raw<0>(d.cfg, s, comp_index(d.ce));
        if (w.lo <= ak && ak <= w.hi && w.at(ak) >= d.sv.tlen) {
          if (G > 1) g.sync();
          d.status = ST_END_REACHED; d.status_score = s; d.end_k = ak;
          return 1;
        }
      }
      *max_ak_out = d.ts.akr[row_buffer(t)];
      return 0;
    }
    // The one-step functions take over at this row.
    int nn = 0;
    for (int q = s - 1; q > 0 && !(holds_row(q, p) && row_exists(d.cb, row_of(q, p), 0)); --q) ++nn;
    if (G > 1) g.sync();
    d.ts.on = 0;
    d.num_null = nn;
    d.next_phys = row_buffer(t);
    if (G > 1) g.sync();
  }
  return dir_step<G, 0, false>(d, p, s, g, max_ak_out);
}
