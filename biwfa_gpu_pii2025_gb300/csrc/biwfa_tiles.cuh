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
// score at a time -> tiles (and the kernel of biwfa_tile_kernel.cuh): 10,000 pairs of 1 kbp at 5 %
// 7.7 -> 3.2 ms, 20,000 uneven pairs (100 bp - 10 kbp, 1-10 %) 320 -> 64 ms, 48 pairs of 10-20 kbp
// at 12 % 560 -> 73 ms, 200,000 pairs of 150 bp at 2 % 15.4 -> 12.3 ms.
//
// Where the values are exact. WFA2-lib trims each row to its in-bounds cells and keeps
// out-of-bounds I/D cells between them. Out-of-bounds cells arise only from a cell whose offset
// has reached the end of the pattern or of the text ("touches": no further extension possible).
// So up to and including the first touched row all values are in bounds or null, trimming only
// removes nulls, and the rows here equal WFA2-lib's with its nulls (any negative offset is null).
// From the row after it the one-step functions (dir_step) continue from the stored rows.

// Null offset of a row. A row treats nulls as cells: one that it passes on grows by 1 and by the
// matches in the window at the sequences' starts (up to 16), so by at most 17 per row. A search's rows
// number at most half of the largest accepted score (2^26) plus the score scope, so no null becomes
// positive; and twice a null, less a diagonal, still fits 32 bits (WFG_TILE_NULL).
constexpr int kTNull = WFG_TILE_NULL;
constexpr int kTileHalo = 4;
constexpr int kTX = 2, kTO = 4;     // rows back to the mismatch and the gap-opening source
constexpr int kTileMinRing = 256;   // narrowest ring that is worth tiles

// Row of score s (rounded down) and whether s has one. With tm = floor(2^32 / tg) + 1 the product is
// exact while s * tg < 2^32: scores stay below 2^27, and the spacing is at most 31 (gap-linear 31/31,
// the largest within the score scope of 32).
__device__ __forceinline__ int row_of(int s, const Pen& p) { return p.tg == 1 ? s : (int)__umulhi((uint32_t)s, p.tm); }
__device__ __forceinline__ bool holds_row(int s, const Pen& p) { return s == row_of(s, p) * p.tg; }

// Diagonals that can hold a non-null cell in row t of a direction that starts in component cb
// (the rows of all components lie inside; both bounds widen monotonically). LIN: one component, rows
// p.lx (mismatch) and p.lo (gap) back, so a row is at most t / p.lo diagonals wide on each side.
template <bool LIN>
__device__ __forceinline__ int row_hi(int cb, int t, const Pen& p) {
  if (LIN) return p.lo == 1 ? t : (int)__umulhi((uint32_t)t, p.lom);
  return cb == CM ? (t < kTO ? 0 : t - kTO + 1) : cb == CI ? t : max(0, t - kTO - 1);
}
template <bool LIN>
__device__ __forceinline__ int row_lo(int cb, int t, const Pen& p) {
  if (LIN) return -row_hi<true>(cb, t, p);
  return cb == CM ? (t < kTO ? 0 : kTO - 1 - t) : cb == CI ? min(0, kTO + 1 - t) : -t;
}
// Whether component ci (0 M, 1 I, 2 D) of row t exists: some cell of it is not null.
template <bool LIN>
__device__ __forceinline__ bool row_exists(int cb, int t, int ci, const Pen& p) {
  if (t < 0) return false;
  if (LIN) {  // sums of lx and lo (each at most 4, without a common factor): all numbers from 6 on
    if (ci != 0) return false;
    for (int r = t; t < 6 && p.lo > 1 && r >= 0; r -= p.lo)
      if (r % p.lx == 0) return true;
    return t >= 6 || p.lo == 1;
  }
  if (cb == CM) return ci == 0 ? (t >= kTO || t % kTX == 0) : t >= kTO;
  if (ci == 0) return t >= 1;
  return ci == (cb == CI ? 1 : 2) ? true : t >= kTO + 1;
}
__device__ __forceinline__ int row_buffer(int t) { return (t + kTileBufs - 1) % kTileBufs; }

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
  bool gaps;           // I and D go to the ring for every row (else for the last one)
  int lane;
  int lx, lo;          // one-component distances: rows back to the mismatch and the gap source (lx 0: none)
};

// Rows t0+1 .. t0+4 of a tile's diagonals, a.k + off in this lane. Lanes j and 16 + j of ak: the
// largest antidiagonal of row t0+1+j in the lower and the upper half warp; touch: the first of the
// four rows (0-3) where this lane touched, else unchanged. The loop over the rows stays rolled (the
// last four rows' registers rotate by moves): instruction fetch bounds this kernel wherever its code
// does not loop. 10,000 pairs of 1 kbp / 150,000 mixture pairs with the row loop rolled 3.29 / 169 ms,
// unrolled by two 3.80 / 177 ms, by four 4.28 / 210 ms.
template <int C, bool LIN>
__device__ __forceinline__ void tile_pass(const TileArgs& a, const SeqView& sv, int off, bool store, int& ak, int& touch) {
  const int k0 = a.k + off;
  const uint32_t idx = (uint32_t)k0 & a.mask;
  const int p3 = 3 * a.pitch;
  int m[4][C], vi[C], vd[C];
  if (k0 >= a.old_lo && k0 < a.old_hi) {
    #pragma unroll
    for (int j = 0; j < 4; ++j) tile_load<C>(a.old_rows + j * p3 + idx, m[j]);
    if (!LIN) {
      tile_load<C>(a.old_rows + 3 * p3 + a.pitch + idx, vi);
      tile_load<C>(a.old_rows + 3 * p3 + 2 * a.pitch + idx, vd);
    }
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
    int n[C];
    uint32_t x[C];
    if constexpr (LIN) {
      // M = max(M[t-lx] + 1, M[t-lo][k-1] + 1, M[t-lo][k+1]), null beyond its diagonal's end
      int gap[C];
      #pragma unroll
      for (int c = 0; c < C; ++c) gap[c] = a.lo == 1 ? m[3][c] : a.lo == 2 ? m[2][c] : a.lo == 3 ? m[1][c] : m[0][c];
      int left = __shfl_up_sync(kFull, gap[C - 1], 1), right = __shfl_down_sync(kFull, gap[0], 1);
      if (a.first) left = kTNull;
      if (a.last) right = kTNull;
      #pragma unroll
      for (int c = 0; c < C; ++c) {
        const int sub = a.lx == 1 ? m[3][c] : a.lx == 2 ? m[2][c] : a.lx == 3 ? m[1][c] : a.lx == 4 ? m[0][c] : kTNull;
        n[c] = max(max(sub, c == 0 ? left : gap[c > 0 ? c - 1 : 0]) + 1, c == C - 1 ? right : gap[c < C - 1 ? c + 1 : C - 1]);
        if (n[c] > min(sv.tlen, sv.plen + k0 + c)) n[c] = kTNull;
      }
    } else {
      // I = max(M[t-4], I[t-1])[k-1] + 1, D = max(M[t-4], D[t-1])[k+1], M = max(M[t-2] + 1, I, D)
      int fi[C], fd[C];
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
    }
    // First windows of all cells (a null cell reads the sequences' starts).
    #pragma unroll
    for (int c = 0; c < C; ++c) {
      const int pp = max(n[c] + (sv.p0 - k0 - c), sv.p0), tt = max(n[c] + sv.t0, sv.t0);
      const uint32_t wp = (uint32_t)pp >> wsh, wt = (uint32_t)tt >> wsh;
      x[c] = __funnelshift_r(seq_word(sv.pw, wp), seq_word(sv.pw, wp + 1), (uint32_t)pp << sv.bshift) ^
             __funnelshift_r(seq_word(sv.tw, wt), seq_word(sv.tw, wt + 1), (uint32_t)tt << sv.bshift);
    }
    bool ends = false, full = false;
    #pragma unroll
    for (int c = 0; c < C; ++c) {
      const int rem = min(sv.tlen, sv.plen + k0 + c) - n[c];  // to the end of diagonal k0 + c
      const int e = min(x[c] ? (first_set(x[c]) >> sv.bshift) : cpw, rem);
      full |= x[c] == 0;
      ends |= e >= rem && (!LIN || k0 + c == sv.tlen - sv.plen);
      n[c] += e;
    }
    // Matches longer than one window (a null cell has none).
    uint32_t more = 0;
    if (full) {
      #pragma unroll
      for (int c = 0; c < C; ++c) if (x[c] == 0 && n[c] >= 0 && n[c] < min(sv.tlen, sv.plen + k0 + c)) more |= 1u << c;
    }
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
      ends |= cur >= end && (!LIN || k0 + c == sv.tlen - sv.plen);
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
      if (!LIN && (a.gaps || j == 3)) { tile_store<C>(ring + a.pitch, vi); tile_store<C>(ring + 2 * a.pitch, vd); }
    }
    ring += p3;
    if (leafw) {
      tile_store<C>(leaf, n);
      if (!LIN) {
        tile_store<C>(leaf + a.leaf_n, vi);
        tile_store<C>(leaf + 2 * a.leaf_n, vd);
      }
    }
    leaf += (LIN ? 1 : 3) * a.leaf_n;
  }
}

// The tiling of block t0 for L lanes into d.ts: tiles, first diagonal, end of the last tile. One tile
// of 4 L diagonals if they hold all of the rows' cells (the cells beside it are null), else tiles with
// halos. narrow: the last tile has two diagonals per lane. False when the ring does not hold them.
template <bool LIN>
__device__ __forceinline__ bool tile_plan(Dir& d, int t0, int L, const Pen& pen) {
  const int hi = row_hi<LIN>(d.cb, t0 + 4, pen), lo = row_lo<LIN>(d.cb, t0 + 4, pen) & ~3, width = hi - lo + 1;
  int tiles = 1, base = lo;
  bool narrow = width <= 2 * L;
  if (width > 4 * L) {
    tiles = (int)((unsigned)(width + 119) / 120u);
    base = lo - kTileHalo;
    narrow = width - (tiles - 1) * 120 <= 56;
  }
  const int end = base + (tiles - 1) * 120 + (narrow ? 2 : 4) * L;
  d.ts.tiles = tiles; d.ts.base = base; d.ts.end = end; d.ts.narrow = narrow;
  // WFA2-lib prunes edit wavefronts of 1,000 diagonals and more: the one-step function's part
  if (LIN && pen.metric == kMetricEdit && 2 * hi + 1 >= 1000) return false;
  return end - base <= d.cfg.W;
}
// Whether half a warp holds block t0's rows.
template <bool LIN>
__device__ __forceinline__ bool tile_half(int cb, int t0, const Pen& p) {
  return row_hi<LIN>(cb, t0 + 4, p) - (row_lo<LIN>(cb, t0 + 4, p) & ~3) < 64;
}

// Starts a direction over window sv in component cb: row 0 with its extension. Returns its offset,
// or -1 when it touches (then nothing is started).
template <bool LIN>
__device__ __noinline__ int tile_start(Dir& d, const SeqView& sv, int cb, int ce, int lane) {
  const int n = min(sv.plen, sv.tlen);
  int off0 = 0;
  if (cb == CM) {
    const int cpw = 32 >> sv.bshift;
    #pragma unroll 1
    for (; off0 < n; off0 += cpw) {
      const uint32_t x = win32(sv.pw, sv.p0 + off0, sv.bshift) ^ win32(sv.tw, sv.t0 + off0, sv.bshift);
      if (x) { off0 += first_set(x) >> sv.bshift; break; }
    }
  }
  if (off0 >= n) {
    if (!LIN || sv.plen == sv.tlen) return -1;
    off0 = n;  // one component: an end that is not the window's corner is an ordinary cell
  }
  d.sv = sv; d.cb = cb; d.ce = ce;
  d.num_null = 0; d.status = ST_OK; d.status_score = 0; d.end_k = INT_MAX;
  d.ts.on = 1; d.ts.t = 0; d.ts.valid = 0; d.ts.touched = 0;
  d.ts.lo = 0; d.ts.hi = 4;
  d.ts.akr[row_buffer(0)] = cb == CM ? 2 * off0 : 0;
  // rows -3 .. 0 on diagonals 0-3: M in buffers 8-11, I and D of row 0
  if (lane < 6) {
    const int row = lane < 4 ? (8 + lane) * 3 : 11 * 3 + lane - 3;
    const int mine = lane < 3 ? -1 : lane - 3;  // the component of row 0
    *reinterpret_cast<int4*>(d.cfg.rdata + wfg_tile_row(row, d.cfg.pitch)) =
        make_int4(mine == comp_index(cb) ? off0 : kTNull, kTNull, kTNull, kTNull);
  }
  __syncwarp();
  return off0;
}

// Whether block t0 has more than kGapTiles tiles: below that its rows fit the caches anyway. The
// diagonals grow by at most two per row, so no block before kGapFirst has.
constexpr int kGapTiles = 3, kGapFirst = (kGapTiles * 120) / 2 - 12;
__device__ __forceinline__ bool tile_wide(int cb, int t0, const Pen& p) {
  return row_hi<false>(cb, t0 + 4, p) - (row_lo<false>(cb, t0 + 4, p) & ~3) + 1 > kGapTiles * 120;
}
// I and D of rows t0+1 .. t0+3 of a wide block, which its pass did not store: most blocks of a search
// are read again only as the next block's last row, and the rows' footprint and traffic in L2 and
// HBM are half with that alone. The last two blocks before the second phase get them here, from M
// (nothing is extended again). All rows stored -> this, on one GB300: 150,000 mixture pairs 160-164 ->
// 152-154 ms (L2 hits 37 % of the rows' sectors before), 20,000 uneven pairs 68.6 -> 64.2 ms, scores only
// of 10,000 pairs of 200 bp - 5 kbp 6.25 -> 5.90 ms; 1 kbp pairs, never as wide, are equal.
__device__ __noinline__ void tile_gaps(const Dir& d, int t0, const Pen& p, int lane) {
  const int lo = row_lo<false>(d.cb, t0 + 4, p) & ~3, hi = row_hi<false>(d.cb, t0 + 4, p);
  const int old_lo = row_lo<false>(d.cb, t0, p) & ~3, old_hi = (row_hi<false>(d.cb, t0, p) + 4) & ~3;
  const int b = (t0 >> 2) % 3, pitch = d.cfg.pitch;
  const int32_t* old_rows = d.cfg.rdata + wfg_tile_row((b == 0 ? 2 : b - 1) * 12, pitch);
  int32_t* new_rows = d.cfg.rdata + wfg_tile_row(b * 12, pitch);
  #pragma unroll 1
  for (int base = lo - 4; base < hi; base += 120) {  // a halo of four diagonals per side
    const int k = base + lane * 4;
    const uint32_t idx = (uint32_t)k & ((uint32_t)d.cfg.W - 1u);
    int vi[4], vd[4], m[4];
    #pragma unroll
    for (int c = 0; c < 4; ++c) vi[c] = vd[c] = m[c] = kTNull;
    const bool in = k >= old_lo && k < old_hi;
    if (in) {
      tile_load<4>(old_rows + 10 * pitch + idx, vi);
      tile_load<4>(old_rows + 11 * pitch + idx, vd);
    }
    #pragma unroll 1
    for (int j = 0; j < 3; ++j) {
      if (in) tile_load<4>(old_rows + j * 3 * pitch + idx, m);
      int fi[4], fd[4];
      #pragma unroll
      for (int c = 0; c < 4; ++c) { fi[c] = max(m[c], vi[c]); fd[c] = max(m[c], vd[c]); }
      int left = __shfl_up_sync(kFull, fi[3], 1), right = __shfl_down_sync(kFull, fd[0], 1);
      if (lane == 0) left = kTNull;
      if (lane == 31) right = kTNull;
      #pragma unroll
      for (int c = 0; c < 4; ++c) { vi[c] = (c == 0 ? left : fi[c > 0 ? c - 1 : 0]) + 1; vd[c] = c == 3 ? right : fd[c < 3 ? c + 1 : 3]; }
      if (lane > 0 && lane < 31 && k <= hi) {
        tile_store<4>(new_rows + (j * 3 + 1) * pitch + idx, vi);
        tile_store<4>(new_rows + (j * 3 + 2) * pitch + idx, vd);
      }
    }
  }
  __syncwarp();
}

// Descriptors of the scores from .. s from their rows (a score without a row is absent).
template <bool LIN>
__device__ __noinline__ void tile_describe(Dir& d, int s, int from, const Pen& p) {
  const DirCfg c = d.cfg;
  #pragma unroll 1
  for (int q = max(from, 0); q <= s; ++q) {
    const int slot = slot_of(c, q), t = row_of(q, p);
    const bool row = holds_row(q, p);
    const int lo = row_lo<LIN>(d.cb, t, p), hi = row_hi<LIN>(d.cb, t, p);
    #pragma unroll 1
    for (int ci = 0; ci < 3; ++ci)
      c.rdesc[slot * 3 + ci] = row && row_exists<LIN>(d.cb, t, ci, p) ? make_int2(lo, hi) : make_int2(kAbsent, INT_MIN);
    c.rphys[slot] = row_buffer(t);
  }
  __syncwarp();
}

// Step of a direction to score s with its descriptors: from the rows computed ahead or, when these
// end, by dir_step. Returns as dir_step.
template <bool LIN>
__device__ __noinline__ int tile_advance(Dir& d, const Pen& p, int s, const Grp<1> g, int* max_ak_out) {
  *max_ak_out = 0;
  if (d.ts.on) {
    const bool row = holds_row(s, p);
    const int t = row_of(s, p);
    if (!row || t <= d.ts.valid) {
      tile_describe<LIN>(d, s, s, p);
      if (!row) return 0;
      if (d.ts.touched && t == d.ts.valid) {
        const int ak = d.sv.tlen - d.sv.plen;
        const WfRef m = ref_raw<0>(d.cfg, s, comp_index(d.ce));
        if (m.lo <= ak && ak <= m.hi && m.at(ak) >= d.sv.tlen) {
          d.status = ST_END_REACHED; d.status_score = s; d.end_k = ak;
          __syncwarp();
          return 1;
        }
      }
      *max_ak_out = d.ts.akr[row_buffer(t)];
      return 0;
    }
    // The one-step functions take over at this row.
    int nn = 0;
    for (int q = s - 1; q > 0 && !(holds_row(q, p) && row_exists<LIN>(d.cb, row_of(q, p), 0, p)); --q) ++nn;
    __syncwarp();
    d.ts.on = 0;
    d.num_null = nn;
    d.next_phys = row_buffer(t);
    __syncwarp();
  }
  return dir_step<1, 0, false>(d, p, s, g, max_ak_out);
}

// The leaf store of a leaf whose rows come in tiles (layout and sizes: wfg_tile_leaf_at): block b's rows
// of leaf_n(b) diagonals from leaf_lo(cb, b) at leaf_at(b) cover row_lo .. row_hi. So a row's place
// follows from its number, without a descriptor.
template <bool LIN>
__device__ __forceinline__ int leaf_q(int b, const Pen& p) { return LIN ? row_hi<true>(CM, b, p) : b; }  // LIN: b / lo
template <bool LIN>
__device__ __forceinline__ int leaf_n(int b, const Pen& p) { return wfg_tile_leaf_n(LIN, leaf_q<LIN>(b, p)); }
template <bool LIN>
__device__ __forceinline__ int leaf_lo(int cb, int b, const Pen& p) {
  return !LIN && cb == CI ? -4 * b : -4 * leaf_q<LIN>(b, p) - 4;
}
template <bool LIN>
__device__ __forceinline__ int leaf_at(int b, const Pen& p) { return wfg_tile_leaf_at(LIN, b, leaf_q<LIN>(b, p), p.lo); }
// Row t's component ci on diagonal k (t >= 1).
template <bool LIN>
__device__ __forceinline__ int leaf_cell(int cb, int t, int ci, int k, const Pen& p) {
  const int b = (t - 1) >> 2, j = (t - 1) & 3;
  return leaf_at<LIN>(b, p) + (LIN ? j : j * 3 + ci) * leaf_n<LIN>(b, p) + k - leaf_lo<LIN>(cb, b, p);
}

// Leaf descriptors of the scores from .. s, for the one-step functions.
template <bool LIN>
__device__ __noinline__ void leaf_describe(Dir& d, int s, int from, const Pen& p, int lane) {
  const int q = max(from, 0) + lane;
  if (q <= s) {
    const int t = row_of(q, p), b = (t - 1) >> 2;
    #pragma unroll 1
    for (int ci = 0; ci < 3; ++ci) {
      int4 ds = make_int4(kAbsent, INT_MIN, 0, 0);
      if (holds_row(q, p) && row_exists<LIN>(d.cb, t, ci, p))
        ds = t == 0 ? make_int4(0, 0, 0, 0)
                    : make_int4(row_lo<LIN>(d.cb, t, p), row_hi<LIN>(d.cb, t, p),
                                leaf_cell<LIN>(d.cb, t, ci, leaf_lo<LIN>(d.cb, b, p), p), leaf_lo<LIN>(d.cb, b, p));
      d.cfg.ldesc[q * 3 + ci] = ds;
    }
  }
  __syncwarp();
}

// leaf_backtrace over a leaf whose rows up to score `fast` came in tiles (later ones
// have descriptors): a lane per source (0 mismatch, 1-2 I open/extend, 3-4 D open/extend), one
// offset latency a step, and the packed maximum picks the source.
// The one-component form gets the penalties by value: a step finds its cell's place from the gap's rows,
// which it would read from shared memory each time (20,000 uneven edit pairs 7.62 -> 7.44 ms); the
// gap-affine form reads them seldom (200,000 pairs of 150 bp 10.25 ms, by value 10.30).
template <bool LIN> struct PenArg { typedef const Pen& type; };
template <> struct PenArg<true> { typedef const Pen type; };
template <bool LIN>
__device__ __noinline__ int tile_backtrace(const Dir& B, typename PenArg<LIN>::type p, int s, int fast, RunOut& out,
                                           uint32_t* lruns, int lruns_cap, int lane) {
  const int cb = B.cb;
  const int32_t* ldata = B.cfg.ldata;
  const int plen = B.sv.plen, tlen = B.sv.tlen;
  const bool ext = lane == 2 || lane == 4, del = lane >= 3;
  const int open = LIN ? p.o : p.o + p.e, back = lane == 0 ? p.x : ext ? p.e : open;
  const bool usable = LIN ? (lane == 0 ? p.metric != kMetricIndel : lane == 1 || lane == 3) : lane < 5;
  const int my_ci = ext ? (del ? 2 : 1) : 0, my_dk = lane == 0 ? 0 : del ? 1 : -1, my_add = del ? 0 : 1;
  const int my_type = lane == 0 ? BT_M : del ? (ext ? BT_D_EXT : BT_D_OPEN) : (ext ? BT_I_EXT : BT_I_OPEN);
  int ci = comp_index(B.ce), score = s, k = B.end_k, off = tlen, nrev = 0, rop = -1, rlen = 0;
  bool over = false;
  int left = plen + tlen + 8;
  // A step's match and its operation, then the start's match and gaps; the last push stores the
  // open run.
  int tail = 0;
  #pragma unroll 1
  for (;;) {
    int eq = 0, op = -2, len = 1;
    if (tail == 0) {
      int mine = INT_MIN;
      bool walk = off - k > 0 && off > 0 && score > 0;
      if (walk) {
        if (--left < 0) return WFG_ST_UNATTAINABLE;
        const int sc = score - back, kk = k + my_dk;
        if (usable && sc >= 0 && (ci == 0 || (lane > 0 && del == (ci == 2)))) {
          int o = kTNull;
          if (sc > fast) {
            o = ref_raw<1>(B.cfg, sc, my_ci).get(kk);
          } else {
            const int t = row_of(sc, p);
            const int at = t == 0 ? (my_ci == comp_index(cb) ? 0 : -1) : leaf_cell<LIN>(cb, t, my_ci, kk, p);
            if (sc == t * p.tg && row_lo<LIN>(cb, t, p) <= kk && kk <= row_hi<LIN>(cb, t, p) && at >= 0) o = ldata[at];
          }
          if (o >= 0) mine = (o + my_add) * 16 + my_type;
        }
        const int best = __reduce_max_sync(kFull, mine);
        walk = best >= 0;
        if (walk && ci == 0) {
          eq = off - (best >> 4);
          off = best >> 4;
          walk = off - k > 0 && off > 0;
        }
        if (walk) {
          const int type = best & 15;
          const bool e = type == BT_I_EXT || type == BT_D_EXT, d = type == BT_D_EXT || type == BT_D_OPEN;
          score -= type == BT_M ? p.x : e ? p.e : open;
          ci = e ? (d ? 2 : 1) : 0;
          op = type == BT_M ? WFG_OP_X : d ? WFG_OP_DEL : WFG_OP_INS;
          if (type != BT_M) k += d ? 1 : -1;
          if (!d) --off;
        }
      }
      if (!walk) { tail = 1; len = 0; }
    } else {
      const int v = off - k, h = off, nm = v > 0 && h > 0 ? min(v, h) : 0;
      if (ci != 0 && (v != 0 || h != 0 || score != 0)) return WFG_ST_UNATTAINABLE;  // WFA2 aborts here
      if (tail == 1) { eq = nm; op = WFG_OP_DEL; len = v - nm; }
      if (tail == 2) { op = WFG_OP_INS; len = h - min(max(v, 0), h); }
      ++tail;
    }
    #pragma unroll 1
    for (int x = 0; x < 2; ++x) {
      const int o = x == 0 ? WFG_OP_EQ : op, n = x == 0 ? eq : len;
      if (n <= 0 && !(x == 1 && tail == 4)) continue;
      if (o == rop) { rlen += n; continue; }
      if (rlen > 0) {
        if (nrev < lruns_cap) lruns[nrev] = ((uint32_t)rlen << 4) | (uint32_t)rop; else over = true;
        ++nrev;
      }
      rop = o; rlen = n;
    }
    if (tail == 4) break;
  }
  if (over) return WFG_ST_SCRATCH_OVERFLOW;
  __syncwarp();
  out.append(lruns, nrev, lane, 32);
  return ST_OK;
}

// wavefront_bialign_overlap over untouched rows: row s0 of d0 against the rows of scores s1,
// s1 - 1, ... of d1. Cells meet where their antidiagonals add up to plen + tlen or more, so the
// lanes first test the rows' largest ones, a row pair each, and only pairs that pass are scanned.
// An untouched row's I and D offsets are at most M's on the same diagonal, so a scan reads M and
// looks at D and I only where M meets. D comes first, then I, then M, the lowest diagonal of each.
template <bool LIN>
__device__ __noinline__ void tile_overlap(const Dir& d0, const Dir& d1, int s0, int s1, bool fwd, BP& bp, const Pen& p,
                                          int lane) {
  const int t0 = row_of(s0, p), cb0 = d0.cb, cb1 = d1.cb;
  if (!row_exists<LIN>(cb0, t0, 0, p)) return;
  const int plen = d0.sv.plen, tlen = d0.sv.tlen, A = tlen - plen;
  const int mine = s1 - lane;
  unsigned todo = __ballot_sync(kFull, lane < p.scope && mine >= 0 && holds_row(mine, p) &&
                                           d0.ts.akr[row_buffer(t0)] + d1.ts.akr[row_buffer(row_of(max(mine, 0), p))] >=
                                               plen + tlen);
  const uint32_t mask = (uint32_t)d0.cfg.W - 1u;
  const int pitch = d0.cfg.pitch;
  const int32_t* r0 = d0.cfg.rdata + wfg_tile_row(row_buffer(t0) * 3, pitch);
  while (todo) {
    const int s = s1 - (__ffs((int)todo) - 1);
    todo &= todo - 1;
    if (s0 + s - p.go >= bp.score) continue;
    const int t1 = row_of(s, p);
    const int32_t* r1 = d1.cfg.rdata + wfg_tile_row(row_buffer(t1) * 3, pitch);
    const int end = min(row_hi<LIN>(cb0, t0, p), A - row_lo<LIN>(cb1, t1, p));
    int first[3] = {INT_MAX, INT_MAX, INT_MAX};  // lowest diagonal where M, I, D meet
    #pragma unroll 1
    for (int kb = max(row_lo<LIN>(cb0, t0, p), A - row_hi<LIN>(cb1, t1, p)) + lane; kb - lane <= end; kb += 128) {
      // four diagonals per lane, their loads in flight together
      int sum[4];
      sum[0] = kb <= end ? r0[(uint32_t)kb & mask] + r1[(uint32_t)(A - kb) & mask] : -1;
      sum[1] = sum[2] = sum[3] = -1;
      if (kb - lane + 32 <= end) {
        #pragma unroll
        for (int u = 1; u < 4; ++u) {
          const int k = kb + 32 * u;
          sum[u] = k <= end ? r0[(uint32_t)k & mask] + r1[(uint32_t)(A - k) & mask] : -1;
        }
      }
      #pragma unroll 1
      for (int u = 0, k = kb; max(max(sum[0], sum[1]), max(sum[2], sum[3])) >= tlen && u < 4; ++u, k += 32) {
        if (sum[0] >= tlen) {
          const uint32_t i0 = (uint32_t)k & mask, i1 = (uint32_t)(A - k) & mask;
          first[0] = min(first[0], k);
          if (!LIN && r0[pitch + i0] + r1[pitch + i1] >= tlen) first[1] = min(first[1], k);
          if (!LIN && r0[2 * pitch + i0] + r1[2 * pitch + i1] >= tlen) first[2] = min(first[2], k);
        }
        sum[0] = sum[1]; sum[1] = sum[2]; sum[2] = sum[3]; sum[3] = -1;
      }
    }
    #pragma unroll
    for (int i = 0; i < 3; ++i) first[i] = __reduce_min_sync(kFull, first[i]);
    const int ci = first[2] != INT_MAX ? 2 : first[1] != INT_MAX ? 1 : 0;
    const int k = ci == 2 ? first[2] : ci == 1 ? first[1] : first[0];
    const int cand = ci ? s0 + s - p.o : s0 + s;
    if (k == INT_MAX || cand >= bp.score) continue;
    const int o0 = r0[ci * pitch + ((uint32_t)k & mask)], o1 = r1[ci * pitch + ((uint32_t)(A - k) & mask)];
    bp.score = cand;
    bp.comp = ci == 2 ? CD : ci == 1 ? CI : CM;
    bp.sf = fwd ? s0 : s; bp.sr = fwd ? s : s0;
    bp.kf = fwd ? k : A - k; bp.kr = fwd ? A - k : k;
    bp.of = fwd ? o0 : o1; bp.orv = fwd ? o1 : o0;
  }
}
