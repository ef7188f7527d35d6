// kernels.cu -- sm_100a kernels of the alignment stage.
//
//  saru_diag_kernel           the production path (reads up to 512 bases, k up
//                             to 15): persistent warps over 32-candidate tiles
//                             (one lane per candidate), furthest columns by
//                             diagonal and error count (diag_tile.cuh),
//                             traceback and slot strings or compact records
//                             on the device; a launch covers segments (calls,
//                             or slices [t0, t1) of one call).
//  saru_full_fill_rows_kernel the exact full-rectangle path for inputs the
//  saru_full_fill_kernel      kernels above do not cover (other costs,
//  saru_full_trace_kernel     m <= 3k, k > 15, irregular windows): the
//                             reference's int16 recurrence over a device
//                             arena holding every matrix of the call (rows in
//                             shared memory; very short and very long reads
//                             cell by cell), then its traceback over that
//                             arena.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>

#include "kernels.cuh"
#include "band_tile.cuh"
#include "diag_tile.cuh"
#include "saru_core.cuh"

namespace saru {

__device__ __forceinline__ long gstart_of(const int32_t *goff, long t) { return t ? goff[t - 1] : 0; }

// ---------------------------------------------------------------------------
// diagonal kernel: persistent warps over warp tiles (diag_tile.cuh)
// ---------------------------------------------------------------------------

__device__ __forceinline__ Quad load_quad(const uint8_t *p) {
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
  return Quad{v.x, v.y, v.z, v.w};
}

// A tile of the launch with its lanes' offsets, loaded while the tile before
// it is aligned.
struct TileAhead {
  int tile, seg;
  int g1, r1, dir;    // the lane's offsets (inclusive) and flag
  int gp, rp;         // lane 0: the offsets before the tile
  int g_lim, r_lim;   // the last offsets of the segment
};

__device__ __forceinline__ long tile_first(const Segment &g, int tile) {
  return g.t0 + 32L * (tile - g.tile_begin);
}

// Starts the loads of a tile (tile < total).
__device__ __forceinline__ void tile_ahead(const KernelArgs &a, int tile, int lane,
                                           TileAhead &x) {
  x.tile = tile;
  int lo = 0, hi = a.nseg - 1;  // last segment with tile_begin <= tile
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.segs[mid].tile_begin <= tile) lo = mid;
    else hi = mid - 1;
  }
  x.seg = lo;
  const Segment &g = a.segs[lo];
  const long t0 = tile_first(g, tile);
  const long t = t0 + lane < g.n ? t0 + lane : g.n - 1;
  x.g1 = g.goff[t];
  x.r1 = g.roff[t];
  x.dir = g.dirs[t];
  x.gp = x.rp = 0;
  if (lane == 0 && t0 > 0) {
    x.gp = g.goff[t0 - 1];
    x.rp = g.roff[t0 - 1];
  }
  x.g_lim = g.goff[g.n - 1];
  x.r_lim = g.roff[g.n - 1];
}

// The byte ranges of a tile whose offsets have arrived.
__device__ __forceinline__ bool tile_span(const KernelArgs &a, const TileAhead &x, int count,
                                          DiagSpan &s) {
  const Segment &g = a.segs[x.seg];
  s.g_lo = __shfl_sync(0xffffffffu, x.gp, 0);
  s.r_lo = __shfl_sync(0xffffffffu, x.rp, 0);
  s.g_hi = __shfl_sync(0xffffffffu, x.g1, 31);
  s.r_hi = __shfl_sync(0xffffffffu, x.r1, 31);
  s.g_lim = x.g_lim;
  s.r_lim = x.r_lim;
  return s.set(g.reads, g.genome, count, g.max_m, g.k);
}

// The whole 16-byte blocks of bytes [lo, hi) of an array to L2.
__device__ __forceinline__ void prefetch_l2(const uint8_t *p, int lo, int hi) {
  const uintptr_t b = ((uintptr_t)(p + lo) + 15) & ~(uintptr_t)15;
  const uintptr_t e = (uintptr_t)(p + hi) & ~(uintptr_t)15;
  if (b < e)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"((uint32_t)(e - b))
                 : "memory");
}

// Starts the copies of a tile's reads and windows to shared memory.
__device__ __forceinline__ void stage_tile(const Segment &g, const DiagSpan &s, Sm reads,
                                           Sm windows, int lane) {
  auto copy16 = [](Sm d, const uint8_t *p) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d.a),
                 "l"(__cvta_generic_to_global(p))
                 : "memory");
  };
  stage_bytes(reads, g.reads, s.r_base, s.r_hi, s.r_lim, lane, copy16, load_quad);
  stage_bytes(windows, g.genome, s.g_base, s.g_hi, s.g_lim, lane, copy16, load_quad);
}

// The lanes' compare parts from the tile's bit streams; the alphabet status
// bit.  eq: row_matches (rows form).
template <class F, bool ODD>
__device__ __forceinline__ int diag_compare(const Segment &g, const DiagSpan &s,
                                            const DiagLayout &D, int lane, Sm slice, DiagLane &l,
                                            uint32_t &eq) {
  int st = 0;
  const Sm sr = slice + D.streams, sw = sr + 12 * D.rw;
  if (ODD) {
    stream_odd(slice, (int)(s.r_hi - s.r_base), sr + 8 * D.rw, lane);
    stream_odd(slice + D.src_r, (int)(s.g_hi - s.g_base), sw + 8 * D.ww, lane);
    __syncwarp();
  }
  const StreamWords R{sr, sr + 4 * D.rw, sr + 8 * D.rw, l.ok ? 32 + (int)(l.rs - s.r_base) : 32};
  const StreamWords W{sw, sw + 4 * D.ww, sw + 8 * D.ww, l.ok ? 32 + (int)(l.gs - s.g_base) : 32};
  const uint8_t *read = g.reads + l.rs, *win = g.genome + l.gs;
  Extras x;
  x.n = 0;
  if (ODD && l.ok && !read_extras(R, D.nr, l.c.m, read, x)) {
    st = 2;  // alphabet
    l.ok = false;
  }
  if (F::ROWS) {
    if (l.ok) eq = lane_rows<ODD>(R, W, l.c, read, win, x, D, RowsOf<F::CUT>(slice, D, lane, g.k));
  } else {
    const Planes<ODD> P(slice, D, lane, g.k);
    lane_planes<ODD>(R, D.nr, l.ok ? l.c.m : 0, read, x, false, P.rd);
    lane_planes<ODD>(W, D.nw, l.ok ? l.c.L : 0, win, x, true, P.wn);
  }
  return st;
}

// Levels and walk of a lane on its mismatch look-up P.
template <typename RW, class X, class Table>
__device__ __forceinline__ int diag_lane(const X &P, const Table &T, RW eq, int reach,
                                         DiagLane &l, WalkEnd &end, const GapMask &U,
                                         const GapMask &Lf) {
  const DiagExit x = lane_levels<RW>(l.c, P, T, eq, reach);
  l.score = x.score;
  if (x.score > T.k) return 0;
  end = lane_diag_walk<RW>(l.c, P, T, x, eq, reach, U, Lf);
  if (!end.bad) return 0;
  end.n = 0;
  return 4;
}

// From the tile's bit streams to the lanes' walks.
template <class F>
__device__ __forceinline__ int diag_align(const Segment &g, const DiagSpan &s, const DiagLayout &D,
                                          bool odd, int lane, Sm slice, DiagLane &l, WalkEnd &end,
                                          const GapMask &U, const GapMask &Lf) {
  constexpr bool ROWS = F::ROWS;
  using RW = typename DiagWord<ROWS>::type;
  uint32_t eq = 0;
  int st = odd ? diag_compare<F, true>(g, s, D, lane, slice, l, eq)
               : diag_compare<F, false>(g, s, D, lane, slice, l, eq);
  __syncwarp();
  const Sm table = slice + D.compare_bytes;
  // table and gap masks (adjacent) start from zero
  for (int i = 16 * lane; i < D.table_bytes + D.masks_bytes; i += 512)
    sm_st128(table + i, Quad{0, 0, 0, 0});
  __syncwarp();
  end = WalkEnd{0, 0, 0, false};
  const DiagTable<F::CELL> T(table, lane, g.k);
  if (!l.ok) return st;
  if (ROWS)
    return st | diag_lane<RW>(RowsOf<F::CUT>(slice, D, lane, g.k), T, (RW)eq, D.reach, l, end, U,
                              Lf);
  const int m = l.c.m;
  if (odd) {
    const Planes<true> P(slice, D, lane, g.k);
    return st | diag_lane<RW>(P, T, (RW)P.matches(m, D.reach), D.reach, l, end, U, Lf);
  }
  const Planes<false> P(slice, D, lane, g.k);
  return st | diag_lane<RW>(P, T, (RW)P.matches(m, D.reach), D.reach, l, end, U, Lf);
}

// One warp tile; `next`: the tile after it (its offsets arrive while this
// one is aligned, its bytes go to L2 while this one's strings are written).
template <class F>
__device__ __forceinline__ int diag_tile(const KernelArgs &a, const TileAhead &now, int next,
                                         TileAhead &ahead, int lane, uint8_t *slice_p, Sm gaps) {
  const Segment &g = a.segs[now.seg];
  const int k = g.k;
  const long t0 = tile_first(g, now.tile);
  const int count = g.n - t0 < 32 ? (int)(g.n - t0) : 32;
  int g0 = __shfl_up_sync(0xffffffffu, now.g1, 1), r0 = __shfl_up_sync(0xffffffffu, now.r1, 1);
  if (lane == 0) {
    g0 = now.gp;
    r0 = now.rp;
  }
  DiagSpan s;
  const bool fits = tile_span(a, now, 32, s);
  DiagLane l;
  int st = lane_candidate(s, g0, now.g1, r0, now.r1, now.dir, k, g.max_m,
                          g.first_of_call && t0 + lane == 0, lane < count, l)
               ? 0
               : 1;
  const DiagLayout D = diag_layout(g.max_m, k, F::ROWS, F::CELL);
  const Sm slice = sm_at(slice_p);
  uint32_t odd = 0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  if (fits) {
    const Sm sr = slice + D.streams, sw = sr + 12 * D.rw;
    odd = stream_planes(slice, (int)(s.r_hi - s.r_base), sr, sr + 4 * D.rw, lane);
    odd |= stream_planes(slice + D.src_r, (int)(s.g_hi - s.g_base), sw, sw + 4 * D.ww,
                         lane);
  }
  const bool more = next < a.total_tiles;
  if (more) tile_ahead(a, next, lane, ahead);
  else ahead.tile = next;
  // the next tile's bytes: to L2 while this one's strings are written, then
  // to shared memory
  DiagSpan sn;
  bool fits_next = false;
  auto prefetch = [&]() {
    if (!more) return;
    fits_next = tile_span(a, ahead, 32, sn);
    if (fits_next && lane == 0) {
      const Segment &h = a.segs[ahead.seg];
      prefetch_l2(h.genome, sn.g_lo, sn.g_hi);
      prefetch_l2(h.reads, sn.r_lo, sn.r_hi);
    }
  };
  auto finish = [&]() {
    if (!more || !fits_next) return;
    const Segment &h = a.segs[ahead.seg];
    const DiagLayout N = diag_layout(h.max_m, h.k, F::ROWS, F::CELL);
    stage_tile(h, sn, slice, slice + N.src_r, lane);
  };
  if (!fits) {  // offsets no regular call can have: report, do not stage
    if (lane < count) g.scores[t0 + lane] = k + 1;
    prefetch();
    finish();
    return 1;
  }
  const Sm masks = slice + (D.compare_bytes + D.table_bytes + 4 * lane);
  const GapMask U{masks}, Lf{masks + D.mwords * 128};
  __syncwarp();
  WalkEnd end;
  const bool any_odd = __any_sync(0xffffffffu, odd != 0);
  st |= diag_align<F>(g, s, D, any_odd, lane, slice, l, end, U, Lf);
  __syncwarp();
  prefetch();
  if (lane < count) g.scores[t0 + lane] = l.score;
  if (g.records) {  // compact records straight to global memory
    if (lane < count) {
      uint32_t *rec = reinterpret_cast<uint32_t *>(g.records + (t0 + lane) * g.rec_bytes);
      const int nwords = (int)(g.rec_bytes >> 2);
      rec[0] = (uint32_t)end.n | (end.bad ? 0x10000u : 0u);
      record_words(end.n, nwords, U, Lf, [&](int w, uint32_t v) { rec[w] = v; });
    }
    // the next tile may be another segment's, whose staged bytes reach over
    // this one's gap masks
    __syncwarp();
    finish();
    return st;
  }
  // the strings: both sources staged again, then one array after the other
  // written over zeros and its slot range copied out
  const Sm out = slice + (D.src_r + D.src_w);
  auto st16 = [](uint8_t *d, const uint8_t *p) {
    *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(p);
  };
  const long s_lo = s.g_lo + k * t0, s_hi = s.g_hi + k * (t0 + count);
  const int slot = l.gs - s.g_lo + k * lane;  // the lane's slot from s_lo
  stage_tile(g, s, slice + 16, slice + (D.src_r + 16), lane);
  for (int pass = 0; pass < 2; ++pass) {
    uint8_t *to = pass ? g.genome_aln : g.read_aln;
    const long o_base = stage_base(to, s_lo);
    for (int i = 16 * lane; i < D.out_bytes; i += 512) sm_st128(out + i, Quad{0, 0, 0, 0});
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (end.n) {
      const int from = pass ? D.src_r + 16 + (int)(l.gs - s.g_base) + end.row
                            : 16 + (int)(l.rs - s.r_base) + end.col;
      expand_masked(out + (slot + (int)(s_lo - o_base)), end.n, slice + from, pass ? Lf : U, gaps);
    }
    __syncwarp();
    stage_out(to, slice_p + (D.src_r + D.src_w), s_lo, s_hi, o_base, lane, st16);
    __syncwarp();
  }
  finish();
  return st;
}

// 16 warps an SM: registers (106 a thread in the rows form, 128 in the planes
// forms) and slices (13.8 KB at 100 bp, k = 5) both end there.  Held to 3 or 5 CTAs of 4 warps: 332 or
// 294 us against 291 for 930k candidates of 100 bp.
constexpr int kDiagCtas = 4;
constexpr int kDiagWarpsPerSm = 4 * kDiagCtas;

// Persistent warps: the first tile of a warp is its own number, later ones
// come from the launch's counter (none: in turn).
template <class F>
__global__ void __launch_bounds__(128, kDiagCtas)
    saru_diag_kernel(const __grid_constant__ KernelArgs a) {
  extern __shared__ uint4 smem_v[];
  __shared__ uint32_t gaps[16];
  if (threadIdx.x < 16) gaps[threadIdx.x] = gap_select((int)threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  uint8_t *slice = reinterpret_cast<uint8_t *>(smem_v) + (long)(threadIdx.x >> 5) * a.warp_smem;
  const int first = (int)(blockIdx.x * warps + (threadIdx.x >> 5));
  if (first >= a.total_tiles) return;
  TileAhead now;
  tile_ahead(a, first, lane, now);
  {
    const Segment &g = a.segs[now.seg];
    const DiagLayout D = diag_layout(g.max_m, g.k, F::ROWS, F::CELL);
    DiagSpan s;
    const Sm raw = sm_at(slice);
    if (tile_span(a, now, 32, s)) stage_tile(g, s, raw, raw + D.src_r, lane);
  }
  while (now.tile < a.total_tiles) {
    int next = now.tile + (int)gridDim.x * warps;
    if (a.counter) {
      if (lane == 0) next = (int)gridDim.x * warps + atomicAdd(a.counter, 1);
      next = __shfl_sync(0xffffffffu, next, 0);
    }
    TileAhead ahead;
    int status = diag_tile<F>(a, now, next, ahead, lane, slice, sm_at(gaps));
    status = __reduce_or_sync(0xffffffffu, status);
    if (status && lane == 0)
      atomicOr(a.segs[now.seg].status,
               (status & 1 ? kStatusIrregular : 0) | (status & 2 ? kStatusAlphabet : 0) |
                   (status & 4 ? kStatusOverflow : 0));
    now = ahead;
  }
}

// ---------------------------------------------------------------------------
// exact full-rectangle path
// ---------------------------------------------------------------------------

__device__ __forceinline__ short min3s(short x, short y, short z) {
  short r = x;
  if (r > y) r = y;
  if (r > z) r = z;
  return r;
}

__global__ void saru_full_fill_kernel(FullArgs a) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  const long gs = gstart_of(a.goff, t), rs = t ? a.roff[t - 1] : 0;
  const long m = a.roff[t] - rs, L = a.goff[t] - gs, W = m + 1;
  int so, eo;
  flank_of(a.dirs[t], a.k, so, eo);
  short *M = a.arena + a.eoff[t];
  const uint8_t *g = a.genome + gs, *r = a.reads + rs;
  for (long j = 0; j <= m; ++j) M[j] = (short)j;
  for (long i = 1; i <= L; ++i) M[i * W] = (short)(i < 2 * so + 1 ? M[(i - 1) * W] : M[(i - 1) * W] + 1);
  for (long i = 0; i < L; ++i) {
    const short *up = M + i * W;
    short *cur = M + (i + 1) * W;
    const uint8_t gi = g[i];
    for (long j = 0; j < m; ++j) {
      const int corr = (j == m - 1 && i >= L - 2 * eo) ? a.mismatch : 0;
      const short d = (short)(up[j] + (gi != r[j] ? a.mismatch : a.match));
      const short l = (short)(cur[j] + a.mismatch);
      const short u = (short)(up[j + 1] + a.mismatch - corr);
      cur[j + 1] = min3s(d, l, u);
    }
  }
  a.scores[t] = M[W * (L + 1) - 1];
}

// The same fill with the row above and the read in shared memory and the
// cells written 16 bytes at a time: a matrix is one run of cells, a lane
// shifts its cells into four registers and stores them at every 8th index of
// the arena.  (The kernel above reads and writes each 2-byte cell in global
// memory, a sector a lane: 631 us for 20k candidates of 36 bp, against 59.)
// Bound by the serial chain along a row, a warp of 32 candidates and
// (m + 1) x 64 + m x 32 bytes of shared memory each.
struct CellRun {
  short *to;     // the next cell
  short *begin;  // the matrix
  uint32_t a[4];
  __device__ __forceinline__ void push(int v) {
    a[0] = fshr32(a[0], a[1], 16);
    a[1] = fshr32(a[1], a[2], 16);
    a[2] = fshr32(a[2], a[3], 16);
    a[3] = __byte_perm(a[3], (uint32_t)v, 0x5432);
    ++to;
    // (a block that begins before the matrix is its head, written apart)
    if (((uintptr_t)to & 15u) == 0 && to - 8 >= begin)
      *reinterpret_cast<uint4 *>(to - 8) = make_uint4(a[0], a[1], a[2], a[3]);
  }
  __device__ __forceinline__ void end() const {  // the cells past the last whole block
    const int left = (int)(((uintptr_t)to >> 1) & 7u);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i >= 8 - left) to[i - 8] = (short)(a[i >> 1] >> (16 * (i & 1)));
  }
};

// Cells whose loads go before their stores (for all the compiler knows, a
// cell's store could be any byte that the next one loads): one by one 74 us
// for the 20k candidates above, four 65, eight 59.
constexpr int kCells = 8;

// PLAIN: no cell can leave 16 bits, so the reference's short arithmetic is
// plain integer arithmetic.
template <bool PLAIN>
__global__ void __launch_bounds__(32) saru_full_fill_rows_kernel(FullArgs a) {
  extern __shared__ uint4 smem_v[];
  short *above = reinterpret_cast<short *>(smem_v) + threadIdx.x;  // column j at 32 * j
  uint8_t *read = reinterpret_cast<uint8_t *>(smem_v) + 64L * (a.max_m + 1) + threadIdx.x;
  const long t = 32L * blockIdx.x + threadIdx.x;
  if (t >= a.n) return;
  const long gs = gstart_of(a.goff, t), rs = t ? a.roff[t - 1] : 0;
  const int m = (int)(a.roff[t] - rs), L = (int)(a.goff[t] - gs);
  int so, eo;
  flank_of(a.dirs[t], a.k, so, eo);
  const uint8_t *g = a.genome + gs;
  for (int j = 0; j < m; ++j) read[32 * j] = a.reads[rs + j];
  auto cut = [](int v) { return PLAIN ? v : (int)(short)v; };
  short *begin = a.arena + a.eoff[t];
  // the matrix's cells before its first 16-byte block lie in row 0, column
  // 0.. (m >= 7) or are written one by one with the whole matrix
  CellRun run{begin, begin, {0, 0, 0, 0}};
  const int head = (int)((8 - (((uintptr_t)begin >> 1) & 7u)) & 7u);
  for (int j = 0; j < head; ++j) begin[j] = (short)j;
  for (int j = 0; j <= m; ++j) {
    above[32 * j] = (short)j;
    run.push(j);
  }
  int first = 0;
  for (int i = 0; i < L; ++i) {
    if (i + 1 >= 2 * so + 1) first = cut(first + 1);
    const uint8_t gi = g[i];
    int left = first, diag = above[0];
    above[0] = (short)first;
    run.push(first);
    auto cell = [&](int j, int up, int base, int corr) {
      const int d = cut(diag + (gi != base ? a.mismatch : a.match));
      const int l = cut(left + a.mismatch);
      const int u = cut(up + a.mismatch - corr);
      left = min(min(d, u), l);
      diag = up;
      above[32 * (j + 1)] = (short)left;
      run.push(left);
    };
    int j = 0;
    for (; j + kCells < m; j += kCells) {
      int up[kCells], base[kCells];
#pragma unroll
      for (int q = 0; q < kCells; ++q) {
        up[q] = above[32 * (j + q + 1)];
        base[q] = read[32 * (j + q)];
      }
#pragma unroll
      for (int q = 0; q < kCells; ++q) cell(j + q, up[q], base[q], 0);
    }
    for (; j < m - 1; ++j) cell(j, above[32 * (j + 1)], read[32 * j], 0);
    // free steps down the last column
    cell(j, above[32 * m], read[32 * j], i >= L - 2 * eo ? a.mismatch : 0);
    if (i == L - 1) a.scores[t] = left;
  }
  run.end();
}

__device__ __forceinline__ short arena_cell(const FullArgs &a, long P) { return a.arena[P]; }

// The reference traceback (src/cuda-functions.cu:108-315) over the arena of
// absolute cells; stops with an overflow flag instead of leaving the slot.
__global__ void saru_full_trace_kernel(FullArgs a) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  if (a.scores[t] > a.k) return;
  const long gs = gstart_of(a.goff, t), rs = t ? a.roff[t - 1] : 0;
  const int m = (int)(a.roff[t] - rs), L = (int)(a.goff[t] - gs), W = m + 1;
  int so, eo;
  flank_of(a.dirs[t], a.k, so, eo);
  const int base = (int)a.eoff[t];  // cell indices fit 32 bits, as in the reference
  const long slot = gs + (long)a.k * t;
  const long slot_end = slot + L + a.k;
  int P = base + (L + 1) * W - 1;
  long ap = slot;
  // the loop bound is on the absolute cell index, as in the reference
  while (P >= W) {
    const short v = arena_cell(a, P);
    short dg, lf, tp;
    if (P % W != 0) {
      dg = arena_cell(a, P - W - 1);
      lf = arena_cell(a, P - 1);
    } else {
      dg = 999;
      lf = 999;
    }
    tp = P != 0 ? arena_cell(a, P - W) : (short)999;
    short width = 0;
    const short width_tmp = (short)((P % W) - 1);
    if (width_tmp > 0) width = width_tmp;
    const short h_tmp = (short)(((P - base - width) / W) - 1);
    const short height = h_tmp > 0 ? h_tmp : 0;
    const int corr =
        ((width == m - 1 && height >= L - 2 * eo) || (so && width == 0 && height <= (so + 1) * 2))
            ? a.mismatch
            : 0;
    const long gi = gs + height, ri = rs + width;
    uint8_t gch = 0, rch = 0;
    if (gi >= 0 && gi < a.genome_bytes) gch = a.genome[gi];
    else atomicOr(a.status, kStatusUndefined);
    if (ri >= 0 && ri < a.read_bytes) rch = a.reads[ri];
    else atomicOr(a.status, kStatusUndefined);
    uint8_t oa, ob;
    int step;
    if (dg + a.mismatch == v) {
      oa = rch; ob = gch; step = W + 1;
    } else if (dg + a.match == v && gch == rch) {
      oa = rch; ob = gch; step = W + 1;
    } else if (tp + a.mismatch - corr == v) {
      oa = '_'; ob = gch; step = W;
    } else if (lf + a.mismatch == v) {
      oa = rch; ob = '_'; step = 1;
    } else {
      break;
    }
    if (ap >= slot_end) {
      atomicOr(a.status, kStatusOverflow);
      break;
    }
    a.read_aln[ap] = oa;
    a.genome_aln[ap] = ob;
    ++ap;
    P -= step;
  }
  for (long i = slot, j = ap - 1; i < j; ++i, --j) {
    uint8_t x = a.read_aln[i]; a.read_aln[i] = a.read_aln[j]; a.read_aln[j] = x;
    x = a.genome_aln[i]; a.genome_aln[i] = a.genome_aln[j]; a.genome_aln[j] = x;
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

constexpr long kMaxCtaSmem = 227 * 1024;  // opt-in shared memory per block on sm_100

// The scratch a caller provides is sized as it always was, by the banded form
// (band_tile.cuh): per lane of a persistent grid, the decision planes of its
// read length.  The diagonal kernel uses the tile counter at its start.
BandLayout band_layout(int max_m, int k, int warps_req, bool wide) {
  const SliceLayout S = slice_layout(max_m, k, wide);
  BandLayout L;
  L.rs_bytes = S.rs_bytes;
  L.ws_bytes = S.ws_bytes;
  L.region_bytes = S.region_bytes;
  L.warp_smem = S.warp_smem;
  long w = kMaxCtaSmem / S.warp_smem;
  L.warps = (int)(w >= 4 ? 4 : (w >= 2 ? 2 : (w >= 1 ? 1 : 0)));
  if (warps_req >= 1 && warps_req < L.warps) L.warps = warps_req;
  L.cta_smem = S.warp_smem * L.warps;
  return L;
}

namespace {
// The opt-in shared-memory limit is an attribute of the kernel on one
// device: set once per device, under a lock, before the first launch there.
std::mutex g_attr_mu;
uint64_t g_attr_done;  // bit d set once device d allows it

cudaError_t allow_smem() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_attr_mu);
  if ((g_attr_done >> dev) & 1u) return cudaSuccess;
  const int attr = cudaFuncAttributeMaxDynamicSharedMemorySize, most = (int)kMaxCtaSmem;
  e = cudaFuncSetAttribute(saru_diag_kernel<DiagForm<true, 1>>, (cudaFuncAttribute)attr,
                             most - 64);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(saru_diag_kernel<DiagForm<true, 1, true>>, (cudaFuncAttribute)attr,
                             most - 64);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(saru_diag_kernel<DiagForm<false, 1>>, (cudaFuncAttribute)attr,
                             most - 64);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(saru_diag_kernel<DiagForm<false, 2>>, (cudaFuncAttribute)attr,
                             most - 64);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(saru_full_fill_rows_kernel<true>, (cudaFuncAttribute)attr, most);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(saru_full_fill_rows_kernel<false>, (cudaFuncAttribute)attr, most);
  if (e == cudaSuccess) g_attr_done |= 1ull << dev;
  return e;
}
}  // namespace

// The largest slice a launch's segments need (the longest reads and the
// largest k may be different segments').
long diag_slice(const KernelArgs &a, bool rows) {
  const int cell = a.max_m <= kByteColumns ? 1 : 2;
  long most = 0;
  for (int i = 0; i < a.nseg; ++i) {
    const long s = diag_layout(a.segs[i].max_m, a.segs[i].k, rows, cell).slice;
    if (s > most) most = s;
  }
  return most;
}

// Whether a launch looks its mismatches up in rows: one word has a bit per
// diagonal -k .. 5k/2 up to k = 9, the columns that a row is looked up at (up to
// m + k) must fit a byte, and the slice must leave room for enough warps.  Rows take 65 us where planes take 73 for 176k candidates of
// 100 bp at k = 5 (slices of 13.8 and 12.0 KB), 66 against 47 for 41k of 133 bp
// at k = 8 (27.9 KB against 15.9).
constexpr long kRowsSlice = 20 * 1024;
constexpr int kRowsMaxK = 9, kRowsMaxM = 200;
static_assert(kRowsMaxM + kRowsMaxK <= kByteColumns, "a table cell is a byte");
bool diag_rows(const KernelArgs &a) {
  return a.max_k <= kRowsMaxK && a.max_m <= kRowsMaxM && diag_slice(a, true) <= kRowsSlice;
}

// Whether a launch's rows cut columns at m.  An instruction a cell, so only
// launches with a read length that needs it do: cut everywhere, 176k
// candidates of 100 bp take 62.7 us instead of 62.2, 930k 281.9 instead of 279.9.
// (Rows long enough for column m + k instead: 120k of 94 bp at k = 6 67.6 us
// against 55.3 cut, of 158 bp at k = 6 91.6 against 84.0.)
bool diag_cut(const KernelArgs &a) {
  for (int i = 0; i < a.nseg; ++i)
    if (columns_cross(a.segs[i].max_m, a.segs[i].k)) return true;
  return false;
}

// CTAs of w warps (shared memory w slices) an SM holds.
int diag_ctas_per_sm(int w, long slice, int smem_per_sm) {
  const long by_smem = smem_per_sm / (w * slice + 64 + 1024);
  const long by_regs = kDiagWarpsPerSm / w;
  return (int)(by_smem < by_regs ? by_smem : by_regs);
}

// Warps per CTA: what was asked for, else the count that keeps the most
// warps on an SM (large slices: CTAs of one warp pack best).
int diag_warps(long slice, int warps_req, int smem_per_sm) {
  const int most = (int)((kMaxCtaSmem - 64) / slice);
  if (warps_req >= 1) return warps_req < most ? warps_req : most;
  int best = 0, warps = 1;
  for (int w = most < 4 ? most : 4; w >= 1; --w) {
    const int n = w * diag_ctas_per_sm(w, slice, smem_per_sm);
    if (n > best) {
      best = n;
      warps = w;
    }
  }
  return warps;
}

// Launches of up to this many tiles a warp take them in turn (no counter to
// clear and to wait for): 176k candidates of 100 bp (2.3 tiles a warp) 65.4 ->
// 61.6 us, mixed lengths 168 -> 161; at 12 tiles a warp the counter is 1 %
// faster.
constexpr int kStaticRounds = 4;

cudaError_t launch_diag_kernel(KernelArgs &a, int sms, int smem_per_sm, int ctas_cap,
                               cudaStream_t s) {
  if (a.nseg < 1 || a.nseg > kMaxSegs) return cudaErrorInvalidValue;
  cudaError_t e = allow_smem();
  if (e != cudaSuccess) return e;
  const bool rows = diag_rows(a);
  a.warp_smem = diag_slice(a, rows);
  const int warps = diag_warps(a.warp_smem, a.warps_req, smem_per_sm);
  if (warps < 1) return cudaErrorInvalidValue;
  long per_sm = diag_ctas_per_sm(warps, a.warp_smem, smem_per_sm);
  if (per_sm < 1) per_sm = 1;
  if (ctas_cap >= 1 && per_sm > ctas_cap) per_sm = ctas_cap;
  const long ctas = (a.total_tiles + warps - 1) / warps;
  a.grid = ctas < sms * per_sm ? ctas : sms * per_sm;
  if (a.total_tiles <= kStaticRounds * a.grid * warps) {
    a.counter = nullptr;
  } else {
    e = cudaMemsetAsync(a.counter, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  const size_t smem = (size_t)(a.warp_smem * warps);
  const unsigned grid = (unsigned)a.grid, threads = 32 * (unsigned)warps;
  if (rows && diag_cut(a)) saru_diag_kernel<DiagForm<true, 1, true>><<<grid, threads, smem, s>>>(a);
  else if (rows) saru_diag_kernel<DiagForm<true, 1>><<<grid, threads, smem, s>>>(a);
  else if (a.max_m <= kByteColumns)
    saru_diag_kernel<DiagForm<false, 1>><<<grid, threads, smem, s>>>(a);
  else saru_diag_kernel<DiagForm<false, 2>><<<grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

long band_grid(int sms, long n, const BandLayout &L, int smem_per_sm, int ctas_cap) {
  const long per_cta = 32L * (L.warps > 0 ? L.warps : 1);
  const long tiles = (n + per_cta - 1) / per_cta;
  long per_sm = smem_per_sm / (L.cta_smem + 1024);
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 16) per_sm = 16;
  if (ctas_cap >= 1 && per_sm > ctas_cap) per_sm = ctas_cap;
  const long g = (long)sms * per_sm;
  return tiles < g ? (tiles > 0 ? tiles : 1) : g;
}

size_t band_scratch_bytes(long grid, int max_m, int k, bool wide, int warps_req) {
  const BandLayout L = band_layout(max_m, k, warps_req, wide);
  return kCounterBytes + (size_t)grid * 32 * (L.warps > 0 ? L.warps : 1) *
                             (size_t)plane_units(max_m, wide) * kPlaneUnit;
}

cudaError_t launch_full_kernels(const FullArgs &a, cudaStream_t s) {
  const int cta = 128;
  const unsigned grid = (unsigned)((a.n + cta - 1) / cta);
  if (grid == 0) return cudaSuccess;
  // the row above and the read of 32 candidates in shared memory: reads of 7
  // bases (so that a matrix's head lies in row 0) up to 2.4 k (227 KB); others
  // cell by cell in global memory
  cudaError_t e = allow_smem();
  if (e != cudaSuccess) return e;
  const size_t rows = 64 * ((size_t)a.max_m + 1) + 32 * (size_t)a.max_m;
  if (a.min_m >= 7 && rows <= (size_t)kMaxCtaSmem) {
    // no cell leaves 16 bits if m + L + 2 steps of the larger cost do not
    const long cost = std::max({1L, labs((long)a.match), labs((long)a.mismatch)});
    const unsigned warps = (unsigned)((a.n + 31) / 32);
    if (cost * ((long)a.max_m + a.max_L + 2) < 32767)
      saru_full_fill_rows_kernel<true><<<warps, 32, rows, s>>>(a);
    else
      saru_full_fill_rows_kernel<false><<<warps, 32, rows, s>>>(a);
  } else {
    saru_full_fill_kernel<<<grid, cta, 0, s>>>(a);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  saru_full_trace_kernel<<<grid, cta, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace saru
