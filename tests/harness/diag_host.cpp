// Host emulation of the diagonal kernel's tile loop (saru_diag_kernel in
// saruman_b200/csrc/kernels.cu) over diag_tile.cuh, for CPU tests: the phases
// run lane by lane in the order the kernel's warp barriers impose, in a
// shared slice of exactly the kernel's size, so that AddressSanitizer sees
// every index that leaves it.  Test infrastructure only.
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "../../saruman_b200/csrc/diag_tile.cuh"

using namespace saru;

static Quad load16(const uint8_t *p) {
  Quad q;
  memcpy(&q, p, 16);
  return q;
}

template <typename RW, class X, class Table>
static int lane(const X &P, const Table &T, RW eq, int reach, DiagLane &ls, WalkEnd &end,
                const GapMask &U, const GapMask &Lf) {
  const DiagExit x = lane_levels<RW>(ls.c, P, T, eq, reach);
  ls.score = x.score;
  if (x.score > T.k) return 0;
  end = lane_diag_walk<RW>(ls.c, P, T, x, eq, reach, U, Lf);
  if (!end.bad) return 0;
  end.n = 0;
  return 4;
}

template <class F, bool ODD>
static int align(const TileArgs &a, const DiagSpan &s, const DiagLayout &D, Sm slice,
                 DiagLane *ls, WalkEnd *end, const GapMask *U, const GapMask *Lf) {
  constexpr bool ROWS = F::ROWS;
  using RW = typename DiagWord<ROWS>::type;
  int st = 0;
  RW eq[32] = {};
  const Sm table = slice + D.compare_bytes, sr = slice + D.streams, sw = sr + 12 * D.rw;
  if (ODD)
    for (int i = 0; i < 32; ++i) {
      stream_odd(slice, (int)(s.r_hi - s.r_base), sr + 8 * D.rw, i);
      stream_odd(slice + D.src_r, (int)(s.g_hi - s.g_base), sw + 8 * D.ww, i);
    }
  for (int i = 0; i < 32; ++i) {
    DiagLane &l = ls[i];
    const StreamWords R{sr, sr + 4 * D.rw, sr + 8 * D.rw, l.ok ? 32 + (int)(l.rs - s.r_base) : 32};
    const StreamWords W{sw, sw + 4 * D.ww, sw + 8 * D.ww, l.ok ? 32 + (int)(l.gs - s.g_base) : 32};
    Extras x;
    x.n = 0;
    if (ODD && l.ok && !read_extras(R, D.nr, l.c.m, a.reads + l.rs, x)) {
      st |= 2;
      l.ok = false;
    }
    const int m = l.ok ? l.c.m : 0, L = l.ok ? l.c.L : 0;
    if (ROWS) {
      const MismatchRows M(slice, D, i, a.k);
      if (l.ok)
        eq[i] = lane_rows<ODD>(R, W, l.c, a.reads + l.rs, a.genome + l.gs, x, D, M);
    } else {
      const Planes<ODD> P(slice, D, i, a.k);
      lane_planes<ODD>(R, D.nr, m, a.reads + l.rs, x, false, P.rd);
      lane_planes<ODD>(W, D.nw, L, a.genome + l.gs, x, true, P.wn);
    }
  }
  memset(table.a, 0, (size_t)(D.table_bytes + D.masks_bytes));
  for (int i = 0; i < 32; ++i) {
    end[i] = WalkEnd{0, 0, 0, false};
    if (!ls[i].ok) continue;
    const DiagTable<F::CELL> T(table, i, a.k);
    const MismatchRows M(slice, D, i, a.k);
    const Planes<ODD> P(slice, D, i, a.k);
    st |= ROWS ? lane<RW>(M, T, eq[i], D.reach, ls[i], end[i], U[i], Lf[i])
               : lane<RW>(P, T, (RW)P.matches(ls[i].c.m, D.reach), D.reach, ls[i], end[i], U[i],
                          Lf[i]);
  }
  return st;
}

template <class F>
static int run(const TileArgs &a) {
  const DiagLayout D = diag_layout(a.max_m, a.k, F::ROWS, F::CELL);
  uint8_t *slice_p = (uint8_t *)aligned_alloc(16, (size_t)D.slice);
  memset(slice_p, 0xA5, (size_t)D.slice);
  const Sm slice = sm_at(slice_p);
  uint32_t gaps[16];
  for (int g = 0; g < 16; ++g) gaps[g] = gap_select(g);
  auto st16 = [](uint8_t *g, const uint8_t *d) { memcpy(g, d, 16); };
  int status = 0;
  for (long t0 = a.t0; t0 < a.n; t0 += 32) {
    const int count = a.n - t0 < 32 ? (int)(a.n - t0) : 32;
    DiagSpan s;
    s.r_lo = t0 ? a.roff[t0 - 1] : 0;
    s.g_lo = t0 ? a.goff[t0 - 1] : 0;
    s.r_hi = a.roff[t0 + count - 1];
    s.g_hi = a.goff[t0 + count - 1];
    s.r_lim = a.roff[a.n - 1];
    s.g_lim = a.goff[a.n - 1];
    if (!s.set(a.reads, a.genome, 32, a.max_m, a.k)) {
      for (long t = t0; t < t0 + count; ++t) a.scores[t] = a.k + 1;
      status |= 1;
      continue;
    }
    const Sm sr = slice + D.streams, sw = sr + 12 * D.rw;
    auto copy16 = [](Sm d, const uint8_t *p) { sm_st128(d, load16(p)); };
    auto stage = [&](int at) {
      for (int lane = 0; lane < 32; ++lane) {
        stage_bytes(slice + at, a.reads, s.r_base, s.r_hi, s.r_lim, lane, copy16, load16);
        stage_bytes(slice + (at + D.src_r), a.genome, s.g_base, s.g_hi, s.g_lim, lane, copy16,
                    load16);
      }
    };
    stage(0);
    uint32_t odd = 0;
    DiagLane ls[32];
    WalkEnd end[32];
    GapMask U[32], Lf[32];
    for (int lane = 0; lane < 32; ++lane) {
      odd |= stream_planes(slice, (int)(s.r_hi - s.r_base), sr, sr + 4 * D.rw, lane);
      odd |= stream_planes(slice + D.src_r, (int)(s.g_hi - s.g_base), sw,
                           sw + 4 * D.ww, lane);
      const long t = t0 + lane < a.n ? t0 + lane : a.n - 1;
      if (!lane_candidate(s, lane && lane < count ? a.goff[t - 1] : s.g_lo, a.goff[t],
                          lane && lane < count ? a.roff[t - 1] : s.r_lo, a.roff[t], a.dirs[t], a.k,
                          a.max_m, a.first_of_call && t0 + lane == 0, lane < count, ls[lane]))
        status |= 1;
      const Sm masks = slice + (D.compare_bytes + D.table_bytes + 4 * lane);
      U[lane] = GapMask{masks};
      Lf[lane] = GapMask{masks + D.mwords * 128};
    }
    status |= odd ? align<F, true>(a, s, D, slice, ls, end, U, Lf)
                  : align<F, false>(a, s, D, slice, ls, end, U, Lf);
    for (int lane = 0; lane < 32; ++lane) {
      const long t = t0 + lane;
      if (t >= a.n) continue;
      a.scores[t] = ls[lane].score;
      if (!a.records) continue;
      uint32_t *rec = reinterpret_cast<uint32_t *>(a.records + t * a.rec_bytes);
      rec[0] = (uint32_t)end[lane].n | (end[lane].bad ? 0x10000u : 0u);
      record_words(end[lane].n, (int)(a.rec_bytes >> 2), U[lane], Lf[lane],
                   [&](int w, uint32_t v) { rec[w] = v; });
    }
    if (a.records) continue;
    const Sm src_r = slice + 16, src_w = slice + (D.src_r + 16),
             out = slice + (D.src_r + D.src_w);
    stage(16);
    for (int pass = 0; pass < 2; ++pass) {
      memset(out.a, 0, (size_t)D.out_bytes);
      const long s_lo = s.g_lo + a.k * t0, s_hi = s.g_hi + a.k * (t0 + count);
      const long o_base = stage_base(pass ? a.genome_aln : a.read_aln, s_lo);
      for (int lane = 0; lane < 32; ++lane) {
        if (!end[lane].n) continue;
        const long slot = ls[lane].gs + (long)a.k * (t0 + lane);
        if (pass)
          expand_masked(out + (int)(slot - o_base), end[lane].n,
                        src_w + ((int)(ls[lane].gs - s.g_base) + end[lane].row), Lf[lane],
                        sm_at(gaps));
        else
          expand_masked(out + (int)(slot - o_base), end[lane].n,
                        src_r + ((int)(ls[lane].rs - s.r_base) + end[lane].col), U[lane],
                        sm_at(gaps));
      }
      for (int lane = 0; lane < 32; ++lane)
        stage_out(pass ? a.genome_aln : a.read_aln, out.a, s_lo, s_hi, o_base, lane, st16);
    }
  }
  free(slice_p);
  return status;
}

// Aligns candidates t0 .. n - 1 of a call; records (rec_bytes each) instead
// of slot strings when records is given.
extern "C" int diag_align_batch(const uint8_t *genome, const uint8_t *reads, const int *goff,
                                const int *roff, const int8_t *dirs, long n, int k, int max_m,
                                int rows, int first_of_call, long t0, int *scores, uint8_t *ra,
                                uint8_t *ga, uint8_t *records, long rec_bytes) {
  TileArgs a{genome, reads, goff, roff, dirs, n, k, max_m, first_of_call, scores, ra, ga,
             nullptr, 0, 0, 0, 0, records, rec_bytes, t0};
  if (rows) return run<DiagForm<true, 1>>(a);
  return max_m <= kByteColumns ? run<DiagForm<false, 1>>(a) : run<DiagForm<false, 2>>(a);
}
