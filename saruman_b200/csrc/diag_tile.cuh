// diag_tile.cuh -- one warp tile of the diagonal kernel, as phases.
//
// A warp tile is 32 consecutive candidates, one per lane.  Instead of every
// cell of the band, a lane computes for each diagonal d = i - j and each
// number of errors e <= k the furthest column whose cell value is <= e
// (E. Ukkonen, Inf. Control 64, 1985; G. Landau, U. Vishkin, J. Algorithms
// 10, 1989): about (k+1)(2so + k) cells a candidate, each extended along its
// diagonal by comparing 32 bases at a time on 2-bit base planes.  Cell
// values grow by 0 or 1 along a diagonal, so the table answers every
// question the reference's traceback asks about a cell with value <= k
// (saru_core.cuh lists them), and the walk goes from error to error instead
// of from column to column.
//
//   reads, windows --> 2-bit planes of the tile's bytes (one bit stream a
//     plane) --> per-lane plane words --> table of furthest columns, score
//     and exit of the last column --> walk (gap masks by step) --> strings
//     or compact records
//
// The phases are separated by warp barriers in the kernel; written as
// functions of the lane so a host harness can run them lane by lane.
#pragma once
#include <assert.h>
#include <stdint.h>

#include "band_tile.cuh"

namespace saru {

// A table cell holds a column + 1: a byte for reads up to 255 bases, two for
// longer ones.
constexpr int kByteColumns = 255;

// The forms a launch runs in: `rows` or planes (DiagLayout), bytes a cell, and
// whether rows cut columns at m (columns_cross).
template <bool ROWS_, int CELL_, bool CUT_ = false>
struct DiagForm {
  static constexpr bool ROWS = ROWS_;
  static constexpr int CELL = CELL_;
  static constexpr bool CUT = CUT_;
};

struct alignas(16) Quad {
  uint32_t x, y, z, w;
};

// Top 32 bits of (hi:lo) << (s & 31): planes hold position p of a sequence
// in bit 31 - (p & 31) of word p >> 5, so a window of 32 positions is one
// funnel shift and its first mismatch a count of leading zeros.
SARU_HD uint32_t fshl32(uint32_t hi, uint32_t lo, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  s &= 31;
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
SARU_HD int clz32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
SARU_HD int bfind32(uint32_t x) {  // the highest set bit, -1 for none
#if defined(__CUDA_ARCH__)
  int r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
#else
  return x ? 31 - __builtin_clz(x) : -1;
#endif
}
SARU_HD int ctz32(uint32_t x) {  // x != 0
#if defined(__CUDA_ARCH__)
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}
SARU_HD uint32_t bitrev32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __brev(x);
#else
  uint32_t r = 0;
  for (int i = 0; i < 32; ++i) r |= ((x >> i) & 1u) << (31 - i);
  return r;
#endif
}
// N shifted up by one, the sign of x entering at the bottom.
SARU_HD uint32_t push_sign(uint32_t N, int x) { return fshl32(N, (uint32_t)x, 1u); }
SARU_HD uint64_t push_sign(uint64_t N, int x) {
  const uint32_t lo = (uint32_t)N, hi = (uint32_t)(N >> 32);
  return (uint64_t)fshl32(hi, lo, 1u) << 32 | fshl32(lo, (uint32_t)x, 1u);
}
// Sum of the four byte products of a and b, added to c.
SARU_HD uint32_t dot4(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  return __dp4a(a, b, c);
#else
  for (int i = 0; i < 4; ++i) c += ((a >> (8 * i)) & 255u) * ((b >> (8 * i)) & 255u);
  return c;
#endif
}

// A place in the warp's shared slice: a 32-bit shared address on the device,
// so that address arithmetic takes one register (through 64-bit pointers the
// levels took twice the instructions), a pointer in the host emulation.
struct Sm {
#if defined(__CUDA_ARCH__)
  uint32_t a;
#else
  uint8_t *a;
#endif
  SARU_HD Sm operator+(int o) const { return Sm{a + o}; }
};
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ Sm sm_at(const void *p) {
  return Sm{(uint32_t)__cvta_generic_to_shared(p)};
}
__device__ __forceinline__ int sm_ld8(Sm p) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(p.a));
  return (int)v;
}
__device__ __forceinline__ int sm_ld16(Sm p) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p.a));
  return (int)v;
}
__device__ __forceinline__ uint32_t sm_ld32(Sm p) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p.a));
  return v;
}
__device__ __forceinline__ Quad sm_ld128(Sm p) {
  Quad q;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
               : "r"(p.a));
  return q;
}
__device__ __forceinline__ void sm_st8(Sm p, int v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(p.a), "r"(v) : "memory");
}
__device__ __forceinline__ void sm_st16(Sm p, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(p.a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sm_st32(Sm p, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(p.a), "r"(v) : "memory");
}
__device__ __forceinline__ void sm_st128(Sm p, Quad q) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(p.a), "r"(q.x), "r"(q.y),
               "r"(q.z), "r"(q.w)
               : "memory");
}
__device__ __forceinline__ void sm_or32(Sm p, uint32_t v) {  // two lanes may own bytes of a word
  asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(p.a), "r"(v) : "memory");
}
__device__ __forceinline__ int sm_low(Sm p, int bits) { return (int)(p.a & (uint32_t)bits); }
#else
inline Sm sm_at(void *p) { return Sm{static_cast<uint8_t *>(p)}; }
inline int sm_ld8(Sm p) { return *p.a; }
inline int sm_ld16(Sm p) { return *reinterpret_cast<uint16_t *>(p.a); }
inline uint32_t sm_ld32(Sm p) { return *reinterpret_cast<uint32_t *>(p.a); }
inline Quad sm_ld128(Sm p) { return *reinterpret_cast<Quad *>(p.a); }
inline void sm_st8(Sm p, int v) {
  assert(v >= 0 && v <= 255);  // a table cell of one byte holds the column
  *p.a = (uint8_t)v;
}
inline void sm_st16(Sm p, uint32_t v) { *reinterpret_cast<uint16_t *>(p.a) = (uint16_t)v; }
inline void sm_st32(Sm p, uint32_t v) { *reinterpret_cast<uint32_t *>(p.a) = v; }
inline void sm_st128(Sm p, Quad q) { *reinterpret_cast<Quad *>(p.a) = q; }
inline void sm_or32(Sm p, uint32_t v) { *reinterpret_cast<uint32_t *>(p.a) |= v; }
inline int sm_low(Sm p, int bits) { return (int)((uintptr_t)p.a & (uintptr_t)bits); }
#endif

SARU_HD int top_bit(uint32_t x) { return 31 - clz32(x); }
SARU_HD int top_bit(uint64_t x) {
  return (x >> 32) ? 63 - clz32((uint32_t)(x >> 32)) : 31 - clz32((uint32_t)x);
}
SARU_HD int low_bit(uint32_t x) { return ctz32(x); }
SARU_HD int low_bit(uint64_t x) {
  return (uint32_t)x ? ctz32((uint32_t)x) : 32 + ctz32((uint32_t)(x >> 32));
}

// ---------------------------------------------------------------------------
// layout of a warp's shared slice
// ---------------------------------------------------------------------------
//
//   [compare: what a lane looks its mismatches up in, see below]
//   [table: 32 cells per diagonal and level, see DiagTable]
//   [gap masks: 2 x mwords x 32 words, and a word more]
// The tile's bytes lie over the front of the first two and their bit streams
// at the end of them until the compare part is made; after the walk the bytes
// come back as the strings' sources, with the output staging behind them.
//
// Two forms of the compare part: `rows`, a lane's mismatch bits of every
// diagonal (a look-up is two words and a shift), and planes, its read's and
// window's 2-bit planes (a look-up compares them: more instructions, but
// the space does not grow with k).

struct DiagLayout {
  int nr, nw;       // words a lane holds of its read / window
  int reach;        // highest diagonal of any level (5k/2), see diag_hi
  int diags;        // rows of mismatches: -k .. reach, an even number of them
  int rw, ww;       // words of one plane's bit stream over the tile's reads / windows
  int mwords;       // words of a gap mask
  int src_r, src_w; // room for the tile's reads and windows
  int out_bytes;    // one output string array of the tile
  int streams;      // where the bit streams lie
  int compare_bytes, table_bytes, masks_bytes, slice;
};

SARU_HD int up16(int x) { return (x + 15) & ~15; }

// Cells before level e in the table: level i holds diagonals -i - 2 .. hi(i)
// + 2 with hi(i) = min(2k + i, 3k - i) (diag_hi at so = eo = k; the next level
// and the walk look at the two beyond on either side).
SARU_HD int table_cells(int e, int k) {
  const int h = k / 2 + 1, x = e < h ? e : h;
  return x * (2 * k + 4 + x) + (e - x) * (3 * k + 5);
}

SARU_HD DiagLayout diag_layout(int max_m, int k, bool rows, int cell) {
  DiagLayout D;
  D.reach = 5 * k / 2;
  D.diags = (k + D.reach + 2) & ~1;
  D.nr = ((max_m + 1) >> 5) + 1;
  D.nw = ((max_m + 2 + D.reach) >> 5) + 1;
  D.rw = max_m + D.nr + 4;
  D.ww = max_m + 2 * k + D.nw + 4;
  D.mwords = ((31 + max_m + 3 * k) >> 5) + 1;
  // 16 bytes before the sources and 48 after them for the word reader
  D.src_r = up16(16 + 16 + 32 * max_m + 48);
  D.src_w = up16(16 + 16 + 32 * (max_m + 2 * k) + 48);
  D.out_bytes = up16(32 * (max_m + 3 * k) + 32);
  D.compare_bytes =
      rows ? (D.diags * D.nr + 2) * 128 : (D.nr + D.nw + 2) * 512;
  const int streams = up16(3 * 4 * (D.rw + D.ww));
  D.table_bytes = table_cells(k > 0 ? k : 1, k) * 32 * cell;
  D.masks_bytes = (2 * D.mwords + 1) * 128;
  int front = D.compare_bytes + D.table_bytes;
  const int raw = D.src_r + D.src_w;
  if (front < raw + D.out_bytes) front = raw + D.out_bytes;
  if (front < raw + streams) front = raw + streams;
  if (front < D.compare_bytes + streams) front = D.compare_bytes + streams;
  D.table_bytes = front - D.compare_bytes;
  D.streams = front - streams;
  D.slice = front + D.masks_bytes;
  return D;
}

// On a diagonal that has reached column m a level's start goes on one column
// past the level before's, so level e looks at column m + e.  Whether such a
// column leaves its diagonal's row (whose words end with the one of column m +
// 1) for the next diagonal's first columns: then columns have to be cut at m.
// Reads shorter than max_m do not cross if max_m does not.
SARU_HD bool columns_cross(int max_m, int k) { return ((max_m + k) >> 5) > ((max_m + 1) >> 5); }

// ---------------------------------------------------------------------------
// planes
// ---------------------------------------------------------------------------

// Bits 1 and 2 of the ASCII code tell A, C, G and T apart.  For a byte that
// is one of them, flipping bits 0 and 4 of T (the one with bit 2 and without
// bit 1) leaves 0x41 with bits 1 and 2 free.
SARU_HD uint32_t acgt_form(uint32_t x) {
  const uint32_t t = x & ~(x << 1) & 0x04040404u;
  return x ^ (t << 2) ^ (t >> 2);
}
// Per byte: 0x80 where the byte is not one of A, C, G, T.
SARU_HD uint32_t not_acgt(uint32_t x) {
  const uint32_t z = (acgt_form(x) ^ 0x41414141u) & 0xF9F9F9F9u;
  return (((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;
}

// A vector of 16 bytes at offset x0 of an array (x0 + array is 16-byte
// aligned); bytes outside [0, lim) of the array are not read and count as A.
template <class Load16>
SARU_HD Quad bytes16(const uint8_t *p, long x0, long lim, Load16 ld16) {
  if (x0 >= 0 && x0 + 16 <= lim) return ld16(p + x0);
  uint32_t v[4];
  for (int w = 0; w < 4; ++w) {
    v[w] = 0;
    for (int i = 0; i < 4; ++i) {
      const long x = x0 + 4 * w + i;
      const uint32_t c = x >= 0 && x < lim ? p[x] : (uint8_t)'A';
      v[w] |= c << (8 * i);
    }
  }
  return Quad{v[0], v[1], v[2], v[3]};
}

// 16 bits (first byte in bit 15) of the byte flags m0..m3, each flag worth
// `unit` in its byte.
SARU_HD uint32_t bits16(uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  const uint32_t hi = dot4(m0, 0x10204080u, dot4(m1, 0x01020408u, 0u));
  const uint32_t lo = dot4(m2, 0x10204080u, dot4(m3, 0x01020408u, 0u));
  return hi * 256u + lo;
}

// The bit streams of `bytes` staged bytes: 16 a step, bit 1 and bit 2 planes
// at s0 / s1 (32-bit words, byte i is position 32 + i).  Returns nonzero if
// a byte is not ACGT (bytes around the tile's, in the edge vectors, count).
// About 50 instructions a step, 14 steps at 100 bp, for check and planes;
// building codes and masks lane by lane took 2.2k.
SARU_HD uint32_t stream_planes(Sm raw, int bytes, Sm s0, Sm s1, int lane) {
  uint32_t any = 0, all = 0xFFFFFFFFu;
  for (int v = lane; 16 * v < bytes; v += 32) {
    const Quad x = sm_ld128(raw + 16 * v);
    const uint32_t f0 = acgt_form(x.x), f1 = acgt_form(x.y), f2 = acgt_form(x.z),
                   f3 = acgt_form(x.w);
    any |= f0 | f1;
    any |= f2 | f3;
    all &= f0 & f1;
    all &= f2 & f3;
    const uint32_t M = 0x02020202u, N = 0x04040404u;
    const int at = 4 + 2 * (v ^ 1);
    sm_st16(s0 + at, bits16(x.x & M, x.y & M, x.z & M, x.w & M) >> 1);
    sm_st16(s1 + at, bits16(x.x & N, x.y & N, x.z & N, x.w & N) >> 2);
  }
  return (any & 0xB8B8B8B8u) | (~all & 0x41414141u);
}

// The stream of the bytes that are not ACGT (tiles that have any).
SARU_HD void stream_odd(Sm raw, int bytes, Sm s2, int lane) {
  for (int v = lane; 16 * v < bytes; v += 32) {
    const Quad q = sm_ld128(raw + 16 * v);
    sm_st16(s2 + (4 + 2 * (v ^ 1)), bits16(not_acgt(q.x) >> 7, not_acgt(q.y) >> 7,
                                           not_acgt(q.z) >> 7, not_acgt(q.w) >> 7));
  }
}

// The bytes [base, hi) of an array (base: stage_base) to dst[0 ..), 16 at a
// time (copy16: an asynchronous copy); bytes outside [0, lim) of the array
// are not read.
template <class Copy16, class Load16>
SARU_HD void stage_bytes(Sm dst, const uint8_t *p, long base, long hi, long lim, int lane,
                         Copy16 copy16, Load16 ld16) {
  const int bytes = (int)(hi - base);
  if (base >= 0 && base + ((hi - base + 15) & ~15L) <= lim) {
    const uint8_t *g = p + base;
    for (int i = 16 * lane; i < bytes; i += 512) copy16(dst + i, g + i);
  } else {
    for (int i = 16 * lane; i < bytes; i += 512)
      sm_st128(dst + i, bytes16(p, base + i, lim, ld16));
  }
}

// 32 positions of a lane's sequence out of the tile's streams: position 1
// of the sequence is stream position `at`.
struct StreamWords {
  Sm s0, s1, s2;
  int at;
  SARU_HD uint32_t from(Sm s, int pos) const {
    const int b = at - 1 + pos;
    const Sm p = s + (b >> 5) * 4;
    return fshl32(sm_ld32(p), sm_ld32(p + 4), (uint32_t)b);
  }
};

// Three plane words of a sequence.
struct Bits3 {
  uint32_t a, b, c;
};
SARU_HD uint32_t differ(const Bits3 &x, const Bits3 &y) {
  return (x.a ^ y.a) | (x.b ^ y.b) | (x.c ^ y.c);
}

// The other bytes than ACGT of a lane's read, by class.
struct Extras {
  uint8_t ch[MAX_EXTRA];
  int n;
};

// Positions p0.. of a sequence.  In a tile with other bytes than ACGT
// (ODD), such a byte gets the class of its byte in the lane's read (the
// first or second distinct one), a window byte that is neither gets a class
// no read byte has, so equality stays byte equality.
template <bool ODD>
SARU_HD Bits3 plane_words(const StreamWords &s, int p0, int len, const uint8_t *bytes,
                          const Extras &x) {
  Bits3 r{s.from(s.s0, p0), s.from(s.s1, p0), 0u};
  if (ODD) {
    r.c = s.from(s.s2, p0);
    for (uint32_t left = r.c; left;) {
      const int z = clz32(left);
      const uint32_t bit = 0x80000000u >> z;
      left &= ~bit;
      const int pos = p0 + z - 1;  // 0-based position in the sequence
      if (pos < 0 || pos >= len) continue;
      int e = 0;
      while (e < x.n && x.ch[e] != bytes[pos]) ++e;
      if (e == x.n) e = 3;
      r.a = (e & 1) ? r.a | bit : r.a & ~bit;
      r.b = (e & 2) ? r.b | bit : r.b & ~bit;
    }
  }
  return r;
}

// The read's other bytes; false if it has more than MAX_EXTRA distinct ones.
SARU_HD bool read_extras(const StreamWords &s, int words, int len, const uint8_t *bytes,
                         Extras &x) {
  x.n = 0;
  for (int w = 0; w < words; ++w) {
    for (uint32_t left = s.from(s.s2, 32 * w); left;) {
      const int z = clz32(left);
      left &= ~(0x80000000u >> z);
      const int pos = 32 * w + z - 1;
      if (pos < 0 || pos >= len) continue;
      int e = 0;
      while (e < x.n && x.ch[e] != bytes[pos]) ++e;
      if (e < x.n) continue;
      if (x.n == MAX_EXTRA) return false;
      x.ch[x.n++] = bytes[pos];
    }
  }
  return true;
}

// Mismatch bits of a lane by diagonal: word w of diagonal d holds columns
// 32w .. (column j, 1-based, is position j; position 0 is padding).  CUT: see
// columns_cross.
template <bool CUT>
struct RowsOf {
  Sm zero;     // diagonal 0
  int stride;  // bytes from a diagonal to the next
  int k;
  typedef Sm Row;
  static constexpr bool kStops = true;  // columns from m on count as mismatches
  static constexpr bool kCut = CUT;
  SARU_HD RowsOf(Sm slice, const DiagLayout &D, int lane, int k_)
      : zero(slice + (k_ * D.nr * 128 + lane * 4)), stride(D.nr * 128), k(k_) {}
  SARU_HD Row row(int d) const { return zero + d * stride; }
  SARU_HD Row next(Row r) const { return r + stride; }
  SARU_HD uint32_t word(int w, Row r) const { return sm_ld32(r + w * 128); }
  // columns s .. s + 31, the first one in the top bit
  SARU_HD uint32_t window(int s, Row r) const {
    const Sm p = r + (s >> 5) * 128;
    return fshl32(sm_ld32(p), sm_ld32(p + 128), (uint32_t)s);
  }
};

using MismatchRows = RowsOf<true>;
using MismatchRowsUncut = RowsOf<false>;

// Columns m and later of word w.
SARU_HD uint32_t past_columns(int m, int w) {
  const int c = 32 * (w + 1) - m;
  return c <= 0 ? 0u : (c >= 32 ? 0xFFFFFFFFu : (1u << c) - 1u);
}

// Diagonals whose last column matches: bit reach - d.
template <bool ODD, class Rows>
SARU_HD uint32_t row_matches(const StreamWords &R, const StreamWords &W, int m, int reach,
                             const Rows &M) {
  if (!ODD) {  // the last read position against window rows m - k ..
    const uint32_t a = 0u - (R.from(R.s0, m) >> 31), b = 0u - (R.from(R.s1, m) >> 31);
    const uint32_t ne = (a ^ W.from(W.s0, m - M.k)) | (b ^ W.from(W.s1, m - M.k));
    return ~ne >> (31 - reach - M.k);
  }
  uint32_t eq = 0;
  Sm p = M.row(-M.k) + (m >> 5) * 128;
  for (int d = -M.k; d <= reach; ++d, p = p + M.stride)
    eq = 2u * eq + (~(sm_ld32(p) << (m & 31)) >> 31);
  return eq;
}

// Fills a lane's rows and returns its row_matches.  Five instructions a
// word: two funnel shifts of the window (its words taken from row -k on, so
// diagonal d is a shift by d + k < 32), two three-input logic operations, a
// store.
template <bool ODD, class Rows>
SARU_HD uint32_t lane_rows(const StreamWords &R, const StreamWords &W, const Cand &c,
                           const uint8_t *read, const uint8_t *win, const Extras &x,
                           const DiagLayout &D, const Rows &M) {
  const int m = c.m, L = c.L, k = M.k;
  Bits3 here = plane_words<ODD>(W, -k, L, win, x);
  for (int w = 0; w < D.nr; ++w) {
    const Bits3 r = plane_words<ODD>(R, 32 * w, m, read, x);
    const Bits3 next = plane_words<ODD>(W, 32 * (w + 1) - k, L, win, x);
    // a level's run ends at column m - 1 at the latest
    const uint32_t past = ODD ? 0u : past_columns(m, w);
    auto one = [&](uint32_t sh) {
      const Bits3 y{fshl32(here.a, next.a, sh), fshl32(here.b, next.b, sh),
                    ODD ? fshl32(here.c, next.c, sh) : 0u};
      return differ(r, y) | past;
    };
    Sm out = M.row(-k) + w * 128;
    for (int sh = 0; sh < D.diags; sh += 2) {
      sm_st32(out, one((uint32_t)sh));
      sm_st32(out + M.stride, one((uint32_t)sh + 1u));
      out = out + 2 * M.stride;
    }
    here = next;
  }
  const uint32_t eq = row_matches<ODD>(R, W, m, D.reach, M);
  if (ODD) {
    for (int w = m >> 5; w < D.nr; ++w) {
      Sm p = M.row(-k) + w * 128;
      for (int d = 0; d < D.diags; ++d, p = p + M.stride)
        sm_st32(p, sm_ld32(p) | past_columns(m, w));
    }
  }
  return eq;
}

// A lane's read and window planes: entry w (16 bytes, 512 bytes apart) holds
// words w and w + 1 of both planes, so 32 positions from any one are one
// load; a tile with other bytes than ACGT keeps three planes a word in
// single words.  The window's entries begin with one for positions -32 ..
// -1 (the walk looks at positions from -k on, whose rows no column has).
template <bool ODD>
struct Planes {
  Sm rd, wn;
  int k;
  typedef int Row;
  static constexpr bool kStops = false;
  static constexpr bool kCut = true;  // entries end with the word of column m + 1
  SARU_HD Planes(Sm slice, const DiagLayout &D, int lane, int k_)
      : rd(slice + lane * 16), wn(slice + (lane * 16 + (D.nr + 1) * 512)), k(k_) {}
  SARU_HD Bits3 bits(Sm seq, int pos) const {
    const Sm p = seq + (pos >> 5) * 512;
    const Quad a = sm_ld128(p);
    const uint32_t sh = (uint32_t)pos;
    if (!ODD) return Bits3{fshl32(a.x, a.y, sh), fshl32(a.z, a.w, sh), 0u};
    const Quad b = sm_ld128(p + 512);
    return Bits3{fshl32(a.x, b.x, sh), fshl32(a.y, b.y, sh), fshl32(a.z, b.z, sh)};
  }
  SARU_HD Row row(int d) const { return d; }
  SARU_HD Row next(Row d) const { return d + 1; }
  SARU_HD uint32_t window(int s, Row d) const { return differ(bits(rd, s), bits(wn, s + d)); }
  SARU_HD uint32_t word(int w, Row d) const { return window(32 * w, d); }
  // diagonals whose last column matches: bit reach - d
  SARU_HD uint64_t matches(int m, int reach) const {
    const Bits3 a = bits(rd, m);
    const Bits3 r{0u - (a.a >> 31), 0u - (a.b >> 31), ODD ? 0u - (a.c >> 31) : 0u};
    const uint32_t hi = ~differ(r, bits(wn, m - k)), lo = ~differ(r, bits(wn, m - k + 32));
    return ((uint64_t)hi << 32 | lo) >> (63 - reach - k);
  }
};

// Fills a lane's plane entries for one sequence (`entries` of them; ODD: one
// more word after them).
template <bool ODD>
SARU_HD void lane_planes(const StreamWords &s, int entries, int len, const uint8_t *bytes,
                         const Extras &x, bool before, Sm out) {
  Bits3 p = plane_words<ODD>(s, 0, len, bytes, x);
  if (!ODD && before) sm_st128(out + -512, Quad{0u, p.a, 0u, p.b});
  for (int w = 0; w < entries; ++w, out = out + 512) {
    const Bits3 q = plane_words<ODD>(s, 32 * (w + 1), len, bytes, x);
    sm_st128(out, ODD ? Quad{p.a, p.b, p.c, 0u} : Quad{p.a, q.a, p.b, q.b});
    p = q;
  }
  if (ODD) sm_st128(out, Quad{p.a, p.b, p.c, 0u});
}

// ---------------------------------------------------------------------------
// furthest columns
// ---------------------------------------------------------------------------

// The table of one lane, levels 0 .. k - 1: at(e, d) is 1 + the furthest
// column of diagonal d with a value <= e, 0 if none is known; columns end at
// m - 1 (the last one has rules of its own).
template <int CELL>
struct DiagTable {
  static constexpr int kStep = 32 * CELL;  // bytes from a diagonal to the next
  Sm base;  // diagonal 0 of level 0
  int k;
  SARU_HD DiagTable(Sm table, int lane, int k_) : base(table + (lane * CELL + 2 * kStep)), k(k_) {}
  SARU_HD Sm cell(int e, int d) const { return base + (table_cells(e, k) + e + d) * kStep; }
  static SARU_HD int get(Sm c) { return CELL == 1 ? sm_ld8(c) : sm_ld16(c); }
  static SARU_HD void put(Sm c, int s) {
    if (CELL == 1) sm_st8(c, s);
    else sm_st16(c, (uint32_t)s);
  }
  SARU_HD int at(int e, int d) const { return get(cell(e, d)); }
  // whether level e has a cell for d
  SARU_HD bool has(int e, int d) const {
    const int hi = 2 * k + e < 3 * k - e ? 2 * k + e : 3 * k - e;
    return d >= -e - 2 && d <= hi + 2;
  }
};

// Diagonals of level e that can still reach the end within k errors: a path
// ends in the last column on diagonals so - eo .. so + eo (free vertical
// moves after that), starts on 0 .. 2so, and changes its diagonal once per
// error at most.
SARU_HD int diag_lo(const Cand &c, int e) {
  const int a = -e, b = c.so - c.eo - (c.k - e);
  return a > b ? a : b;
}
SARU_HD int diag_hi(const Cand &c, int e) {
  const int a = 2 * c.so + e, b = c.so + c.eo + c.k - e;
  return a < b ? a : b;
}

// A word with a bit per diagonal, reach - d for diagonal d of -k .. reach: 32
// bits hold k <= 9, the most the rows form takes.
template <bool ROWS>
struct DiagWord {
  typedef uint32_t type;
};
template <>
struct DiagWord<false> {
  typedef uint64_t type;
};

// Where the traceback leaves the last column.
struct DiagExit {
  int score;  // D[L][m], or k + 1
  int ups;    // UP steps from row L
  int d;      // diagonal of the cell (in column m) it leaves the free rows at
  int how;    // OP_DIAG, OP_LEFT, or OP_UP: on below the free rows
  int v;      // value of the next cell (in column m for OP_UP)
};

// Levels 0 .. k of one lane.  X: its mismatches (RowsOf or Planes);
// eq: the diagonals whose last column matches (RW: bit reach - d).
//
// Bound by instruction issue: about 17 instructions a cell on rows (the
// start from three neighbours, two shared loads, a funnel shift, a count of
// leading zeros, a byte stored), 31 on planes, independent along a level.
// At 100 bp and k = 5 a candidate has 36 cells (so = 0) or 78 against 100
// columns of about 85 instructions (fill, decisions, walk) of the banded
// form.
template <typename RW, class X, class Table>
SARU_HD DiagExit lane_levels(const Cand &c, const X &P, const Table &T, RW eq, int reach) {
  constexpr int N = Table::kStep;
  const int k = c.k, m = c.m;
  DiagExit x;
  x.score = k + 1;
  x.ups = x.d = x.how = x.v = 0;
  // rows L - 2eo .. L of the last column
  const RW ends = lowmask<RW>(reach - c.so + c.eo + 1) & ~lowmask<RW>(reach - c.so - c.eo);
  RW Rp = 0, Vp = 0;  // the level before: diagonals at column m - 1, rows of column m
  for (int e = 0; e <= k; ++e) {
    const int lo = diag_lo(c, e), hi = diag_hi(c, e);
    // level 0 has nothing before it: its own row, read ahead of its writes,
    // is still zero
    Sm prev = T.cell(e > 0 ? e - 1 : 0, lo), cur = T.cell(e, lo);
    typename X::Row row = P.row(lo);
    RW short_of = 0;  // diagonals not at column m - 1 yet, the last one in bit 0
    // from the three neighbours of the level before (diagonals d - 1, d, d +
    // 1): a substitution or a step left goes on one column further, a step
    // up in the same column
    auto start = [](int pm, int p0, int p1) {
      const int s = (p0 > p1 ? p0 : p1) + 1;
      return s > pm ? s : pm;
    };
    // on along the diagonal past the first window of 32 columns (its first
    // mismatch at bit f, -1: none)
    auto extend = [&](int &s, int f, typename X::Row r) {
      while (f < 0 && (X::kStops || s < m)) {
        f = bfind32(P.window(s, r));
        s += 31 - f;
      }
    };
    // (level k is not stored: the walk asks for lower values only)
    auto keep = [&](Sm to, int s) {
      if (X::kCut) s = s < m ? s : m;
      short_of = push_sign(short_of, s - m);
      if (e < k) Table::put(to, s);
    };
    // a level has an odd number of diagonals: one, then fours and a pair, so
    // that one's loads cover the others'
    int pm = Table::get(prev), p0 = Table::get(prev + N);
    {
      int s = start(Table::get(prev + -N), pm, p0);
      const int f = bfind32(P.window(s, row));
      s += 31 - f;
      if (f < 0) extend(s, f, row);
      keep(cur, s);
    }
    int left = hi - lo;
    for (; left >= 4; left -= 4) {
      prev = prev + 4 * N;
      cur = cur + 4 * N;
      const int p1 = Table::get(prev + -2 * N), p2 = Table::get(prev + -N), p3 = Table::get(prev),
                p4 = Table::get(prev + N);
      int sa = start(pm, p0, p1), sb = start(p0, p1, p2), sc = start(p1, p2, p3),
          sd = start(p2, p3, p4);
      const typename X::Row r1 = P.next(row), r2 = P.next(r1), r3 = P.next(r2), r4 = P.next(r3);
      const int fa = bfind32(P.window(sa, r1)), fb = bfind32(P.window(sb, r2)),
                fc = bfind32(P.window(sc, r3)), fd = bfind32(P.window(sd, r4));
      sa += 31 - fa;
      sb += 31 - fb;
      sc += 31 - fc;
      sd += 31 - fd;
      if ((fa | fb | fc | fd) < 0) {
        extend(sa, fa, r1);
        extend(sb, fb, r2);
        extend(sc, fc, r3);
        extend(sd, fd, r4);
      }
      keep(cur + -3 * N, sa);
      keep(cur + -2 * N, sb);
      keep(cur + -N, sc);
      keep(cur, sd);
      pm = p3;
      p0 = p4;
      row = r4;
    }
    if (left) {
      const int p1 = Table::get(prev + 2 * N), p2 = Table::get(prev + 3 * N);
      int sa = start(pm, p0, p1), sb = start(p0, p1, p2);
      const typename X::Row r1 = P.next(row), r2 = P.next(r1);
      const int fa = bfind32(P.window(sa, r1)), fb = bfind32(P.window(sb, r2));
      sa += 31 - fa;
      sb += 31 - fb;
      if ((fa | fb) < 0) {
        extend(sa, fa, r1);
        extend(sb, fb, r2);
      }
      keep(cur + N, sa);
      keep(cur + 2 * N, sb);
    }
    const RW R = (RW)((RW)~short_of & lowmask<RW>(hi - lo + 1)) << (RW)(reach - hi);
    // the last column: a row has value <= e by a diagonal step (a mismatch
    // from e - 1, a match from e), a step left or a step up; steps up are
    // free from row L - 2eo on, so the first level with a row there is the
    // score
    const RW DG = Rp | (R & eq);
    const RW V = DG | (RW)(Rp << 1) | (Vp >> 1);
    const RW hit = V & ends;
    if (hit) {
      x.score = e;
      const RW dg = DG & ends;
      if (dg) {  // the highest row with a diagonal step, free steps up before it
        const int b = low_bit(dg);
        x.d = reach - b;
        x.how = OP_DIAG;
        x.v = ((Rp >> b) & RW(1)) ? e - 1 : e;
      } else {
        const int b = top_bit(hit);
        x.d = reach - b;
        const bool up = x.d == c.so - c.eo && x.d > -k && ((Vp >> (b + 1)) & RW(1));
        x.how = up ? OP_UP : OP_LEFT;
        x.v = e - 1;
      }
      x.ups = c.so + c.eo - x.d;
      break;
    }
    Rp = R;
    Vp = V;
  }
  return x;
}

// ---------------------------------------------------------------------------
// walk
// ---------------------------------------------------------------------------

// The gap steps of one lane's traceback: bit 32 + i of a mask is step i
// (0 at the alignment end); words of a lane 32 apart.
struct GapMask {
  Sm w;
  SARU_HD void add(int i, uint32_t bits) const {
    const Sm p = w + (i >> 5) * 128;
    sm_st32(p, sm_ld32(p) | bits);
  }
  SARU_HD void set(int i) const { add(i + 32, 1u << (i & 31)); }
  SARU_HD void range(int i, int n) const {  // steps i .. i + n - 1 (n <= 64)
    if (n <= 0) return;
    const int b = i & 31;
    add(i + 32, lowmask<uint32_t>(n) << b);
    n -= 32 - b;
    if (n > 0) add(i + 64, lowmask<uint32_t>(n));
    if (n > 32) add(i + 96, lowmask<uint32_t>(n - 32));
  }
  // bits b .. b + 31 of the mask (b >= 0)
  SARU_HD uint32_t window(int b) const {
    const Sm p = w + (b >> 5) * 128;
    return fshr32(sm_ld32(p), sm_ld32(p + 128), (uint32_t)b);
  }
};

// Largest column q <= c of diagonal d whose bytes differ, or something <= 0
// (or below the diagonal's first column, where the planes hold no rows).
template <class X>
SARU_HD int last_mismatch(const X &P, int c, int d) {
  int w = c >> 5;
  const typename X::Row r = P.row(d);
  uint32_t x = P.word(w, r) & (0xFFFFFFFFu << (31 - (c & 31)));
  while (x == 0 && w > 0) x = P.word(--w, r);
  return x ? 32 * w + 31 - ctz32(x) : 0;
}

// Value of row i in column 1 with a free start (so > 0): rows up to 2so + 1
// cost 0 or 1, later ones one more per row, less one once a row from
// 2so + 1 on matches.
template <class X>
SARU_HD int first_column(const X &P, int so, int i) {
  if (i == 0) return 1;
  if (i <= 2 * so + 1) return (int)(P.window(1, P.row(i - 1)) >> 31);
  int v = i - 2 * so;
  for (int r = 2 * so + 1; r <= i; ++r)
    if (!(P.window(1, P.row(r - 1)) >> 31)) return v - 1;
  return v;
}

// The traceback of one lane (the reference's get_alignment,
// src/cuda-functions.cu:108-315) over its table.  On a diagonal, from a cell
// of value v the DIAG step is taken while the bytes match or the cell before
// has value v - 1; so the walk goes straight to the cell after the last
// mismatch (a gap step: UP if the cell above has value v - 1, else LEFT) or
// to the furthest cell of value v - 1, whichever comes first: at most
// 2 v + 1 rounds.  The borders follow the reference's rules (saru_core.cuh,
// traceback_band).
template <typename RW, class X, class Table>
SARU_HD WalkEnd lane_diag_walk(const Cand &c, const X &P, const Table &T, const DiagExit &x,
                               RW eq, int reach, const GapMask &U, const GapMask &Lf) {
  const int m = c.m, so = c.so, k = c.k;
  int nup = x.ups, d = x.d, v = x.v, col = m;
  bool stop = false, bad = false;
  U.range(0, nup);
  int how = x.how;
  if (how == OP_UP) {  // below the free rows of the last column: every step up costs one
    auto at_end = [&](int e, int dd) { return e >= 0 && T.has(e, dd) && T.at(e, dd) >= m; };
    auto diag = [&](int e, int dd) {
      return at_end(e - 1, dd) || (at_end(e, dd) && dd >= -k && ((eq >> (RW)(reach - dd)) & RW(1)));
    };
    U.set(nup++);
    --d;
    for (;;) {
      if (diag(v, d)) {
        how = OP_DIAG;
        if (at_end(v - 1, d)) --v;
        break;
      }
      bool up = false;  // whether the cell above has value v - 1
      for (int e = v - 1, dd = d - 1; e >= 0 && !up; --e, --dd)
        up = diag(e, dd) || at_end(e - 1, dd + 1);
      if (!up) {
        how = OP_LEFT;
        --v;
        break;
      }
      U.set(nup++);
      --d;
      --v;
    }
  }
  if (how == OP_LEFT) {
    Lf.set(nup);
    ++d;
  }
  --col;  // the cell of diagonal d in column m - 1, with value v
  while (col > 0 && col + d > 0) {
    const int lo = d < 0 ? -d : 0;  // the diagonal's cell on row 0 or column 0
    if (v <= 0) {
      col = lo;
      break;
    }
    if (!T.has(v - 1, d) || !T.has(v - 1, d - 1)) {
      bad = true;
      break;
    }
    const int g = T.at(v - 1, d) - 1;
    const int q = last_mismatch(P, col, d);
    if (g >= lo) {
      if (q <= g + 1) {
        col = g;
        --v;
        continue;
      }
    } else if (q <= lo) {
      col = lo;
      break;
    }
    col = q;
    if (so && q == 1) {
      // column 1 with a free start: the step up costs nothing for rows up to
      // 2so + 3
      int i = 1 + d;
      auto start = [&](int r) { return r > 2 * so ? r - 2 * so : 0; };
      for (;;) {
        const bool ne = P.window(1, P.row(i - 1)) >> 31;
        if (start(i - 1) + 1 == v || (start(i - 1) == v && !ne)) {  // DIAG
          --i;
          col = 0;
          break;
        }
        const int tp = first_column(P, so, i - 1);
        if (tp + (i - 1 <= 2 * so + 2 ? 0 : 1) == v) {  // UP
          U.set(m - 1 + nup);
          ++nup;
          v = tp;
          if (--i == 0) break;
          continue;
        }
        if (start(i) + 1 == v) {  // LEFT
          Lf.set(m - 1 + nup);
          col = 0;
        } else {
          stop = true;
        }
        break;
      }
      d = i - col;
      break;
    }
    const bool up = T.at(v - 1, d - 1) > q;
    (up ? U : Lf).set(m - q + nup);
    nup += up;
    d += up ? -1 : 1;
    col -= up ? 0 : 1;
    --v;
  }
  int row = col + d;
  if (!stop && !bad) {
    const int n = m - col + nup;
    if (row == 0) {
      // row 0: the first candidate of a call stops, later ones step left
      if (col > 0 && !c.first_of_call) {
        Lf.range(n, col);
        col = 0;
      }
    } else if (col == 0) {
      // column 0 holds max(0, row - 2so); steps up are taken to row 0, but
      // with a free start not across rows 2so + 1 .. 2so + 3
      int up = row;
      if (so && row > 2 * so) up = row > 2 * so + 3 ? row - (2 * so + 3) : 0;
      U.range(n, up);
      nup += up;
      row -= up;
    }
  }
  const int n = m - col + nup;
  return WalkEnd{n, row, col, bad || n > c.L + k};
}

// ---------------------------------------------------------------------------
// results
// ---------------------------------------------------------------------------

// Entry g of the string writer's table, for four positions of which those in
// g (bit 3: the first) are gaps: a byte selector over (source, '_') in the
// low half, the source bytes used in the high half.
SARU_HD uint32_t gap_select(int g) {
  uint32_t sel = 0;
  int used = 0;
  for (int i = 0; i < 4; ++i) sel |= (uint32_t)((g >> (3 - i)) & 1 ? 4 : used++) << (4 * i);
  return sel | (uint32_t)used << 16;
}

// One alignment string of a lane at dst[0, n) of the zero-filled staging:
// the bytes of src in order with '_' at the gap steps.  Every word of dst's
// word grid takes the next four source bytes and places them by the table
// entry of its four gap bits, so a gap costs no branch; the two edge words,
// which share bytes with the neighbouring slots, are ORed in.  Reads up to 6
// bytes before src and 7 past its end.
SARU_HD void expand_masked(Sm dst, int n, Sm src, const GapMask &G, Sm table) {
  const int a = sm_low(dst, 3);
  Sm to = dst + -a, from = src + -a;
  int left = n + a;  // bytes from the word on; its positions are steps left - 1 downwards
  auto word = [&](uint32_t gap4) -> uint32_t {  // the four gap bits, times 4
    const uint32_t sel = sm_ld32(table + (int)(gap4 & 60u));
    const int low = sm_low(from, 3);
    const Sm p = from + -low;
    const uint32_t v = fshr32(sm_ld32(p), sm_ld32(p + 4), (uint32_t)low * 8u);
    from = from + (int)(sel >> 16);
    return byte_perm(v, 0x5F5F5F5Fu, sel);
  };
  if (a) {
    sm_or32(to, word(G.window(left) >> 26) & bytes_mask(a, left < 4 ? left : 4));
    to = to + 4;
    left -= 4;
  }
  for (; left >= 32; left -= 32, to = to + 32) {
    const uint32_t bits = G.window(left);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      sm_st32(to + 4 * i, word(i < 7 ? bits >> (26 - 4 * i) : bits << 2));
  }
  if (left > 0) {
    uint32_t bits = G.window(left);
    for (; left >= 4; left -= 4, bits <<= 4, to = to + 4) sm_st32(to, word(bits >> 26));
    if (left > 0) sm_or32(to, word(bits >> 26) & bytes_mask(0, left));
  }
}

// 16 bits to the even bits of a word.
SARU_HD uint32_t spread16(uint32_t x) {
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}

// The step words of a compact record from the gap masks, two at a time:
// store(w, v) gets words 1 .. nwords - 1.
template <class Store>
SARU_HD void record_words(int n, int nwords, const GapMask &U, const GapMask &Lf, Store store) {
  for (int w = 1; w < nwords; w += 2) {
    const int lo = 16 * (w - 1);  // the first step of word w
    uint32_t a = 0, b = 0;
    if (lo < n) {
      const uint32_t valid = lowmask<uint32_t>(n - lo);
      const uint32_t u = U.window(lo + 32), g = (u | Lf.window(lo + 32)) & valid, t = valid & ~u;
      a = spread16(t & 0xFFFFu) | spread16(g & 0xFFFFu) << 1;  // DIAG 1, UP 2, LEFT 3
      b = spread16(t >> 16) | spread16(g >> 16) << 1;
    }
    store(w, a);
    if (w + 1 < nwords) store(w + 1, b);
  }
}

// ---------------------------------------------------------------------------
// lane set-up
// ---------------------------------------------------------------------------

// A tile's byte ranges in the call's reads and windows, and where the arrays
// end (nothing past that is read).
struct DiagSpan {
  int r_lo, r_hi, r_lim, g_lo, g_hi, g_lim;
  long r_base, g_base;  // stage_base of the ranges

  // false for ranges regular candidates cannot have: such a tile is not
  // staged at all (its candidates are reported irregular)
  SARU_HD bool set(const uint8_t *reads, const uint8_t *genome, int count, int max_m, int k) {
    r_base = stage_base(reads, r_lo);
    g_base = stage_base(genome, g_lo);
    return r_lo >= 0 && g_lo >= 0 && r_hi >= r_lo && g_hi >= g_lo && r_lim >= r_hi &&
           g_lim >= g_hi && (long)r_hi - r_lo <= (long)count * max_m &&
           (long)g_hi - g_lo <= (long)count * (max_m + 2 * k);
  }
};

// A lane's candidate: its window [gs, gs + L) and read [rs, rs + m).
struct DiagLane {
  Cand c;
  int gs, rs;
  int score;
  bool ok;
};

// Sets up a lane from its candidate's offsets; not ok (and false, unless
// `in` is false: past the call's end) if the layout is not the one the
// reference's caller builds, or lies outside the tile's ranges.
SARU_HD bool lane_candidate(const DiagSpan &s, int g0, int g1, int r0, int r1, int dir, int k,
                            int max_m, bool first, bool in, DiagLane &l) {
  l.score = k + 1;
  l.gs = g0;
  l.rs = r0;
  Cand &c = l.c;
  c.m = r1 - r0;
  c.L = g1 - g0;
  c.k = k;
  flank_of(dir, k, c.so, c.eo);
  c.first_of_call = first;
  l.ok = in && c.L == c.m + c.so + c.eo && c.m > 3 * k && c.m <= max_m && c.m >= 2 &&
         r0 >= s.r_lo && r1 <= s.r_hi && g0 >= s.g_lo && g1 <= s.g_hi;
  return l.ok || !in;
}

}  // namespace saru
