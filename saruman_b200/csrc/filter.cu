// filter.cu -- the q-gram pair filter on the device.
//
//  index    every q-gram of the resident genome, hashed (64-bit FNV-1a of its
//           bytes) and sorted with its position (a stable radix sort keeps
//           each q-gram's positions in genome order, as the reference's
//           index lists them, src/util.c:462-480); equal hashes of unequal
//           q-grams are reported, not trusted.
//  lookup   one thread per (read, q-gram): the q-gram of the strand-adjusted
//           read, its run in the sorted index (a table of the hashes' top bits
//           narrows the search; checked against the genome bytes) and, by an
//           exclusive scan, its list's offset in the reference's data array
//           (lists in q-gram order per read, each followed by a 0,
//           src/hash.c:404-457).
//  filter   one warp per read, reads taken most estimated work first, a lane
//           per position of the first-half q-grams (position_hit,
//           filter_core.cuh); the read's kept positions into its slice of a
//           scratch.
//  calls    the kept positions that are candidates and the perfect hits
//           written back to back on the device (a scan over the reads gives
//           their places), copied out while the next launch runs; the host
//           only sets the call boundaries (filter_calls.h states the rules).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/saruman_b200.h"
#include "filter_core.cuh"
#include "server_internal.h"

namespace {

using namespace saru;

constexpr int kHitsPerRead = 4096;   // kept positions per read and strand
constexpr int kReadsPerLaunch = 1 << 16;

// Sum of the scan over list lengths: 64 bits over 32-bit inputs.
struct AddLong {
  __host__ __device__ long operator()(long a, long b) const { return a + b; }
};

__host__ __device__ inline uint64_t qgram_hash(const uint8_t *p, int q) {
  uint64_t h = 1469598103934665603ull;  // FNV-1a 64
  for (int i = 0; i < q; ++i) {
    h ^= p[i];
    h *= 1099511628211ull;
  }
  return h;
}

__device__ inline uint8_t comp_byte(uint8_t c) {
  switch (c) {
    case 'A': return 'T';
    case 'C': return 'G';
    case 'G': return 'C';
    case 'T': return 'A';
    default: return c;
  }
}

__global__ void k_qgram_hash(const uint8_t *g, long npos, int q, uint64_t *hash, uint32_t *pos) {
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < npos;
       p += (long)gridDim.x * blockDim.x) {
    hash[p] = qgram_hash(g + p, q);
    pos[p] = (uint32_t)p;
  }
}

__global__ void k_index_check(const uint64_t *hash, const uint32_t *pos, long n, const uint8_t *g,
                              int q, int *flag) {
  for (long i = 1 + blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    if (hash[i] != hash[i - 1]) continue;
    const uint8_t *a = g + pos[i], *b = g + pos[i - 1];
    for (int j = 0; j < q; ++j)
      if (a[j] != b[j]) {
        atomicOr(flag, 1);
        break;
      }
  }
}

// byte i of the read as its strand aligns it (reverse complement for dr 4)
__device__ inline uint8_t strand_byte(const uint8_t *read, int m, int dr, int i) {
  return dr == 4 ? comp_byte(read[m - 1 - i]) : read[i];
}

// The first index of every value of the hashes' top bits: bucket[v] ..
// bucket[v + 1] are the hashes with top bits v.
__global__ void k_buckets(const uint64_t *hash, long n, int shift, uint32_t nbuckets,
                          uint32_t *bucket) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i <= n;
       i += (long)gridDim.x * blockDim.x) {
    const uint32_t from = i ? (uint32_t)(hash[i - 1] >> shift) + 1 : 0;
    const uint32_t to = i < n ? (uint32_t)(hash[i] >> shift) : nbuckets;
    for (uint32_t v = from; v <= to; ++v) bucket[v] = (uint32_t)i;
  }
}

struct LookupArgs {
  const uint8_t *reads;  // nreads x m, as sequenced
  long nreads;
  int dr;
  FilterShape S;
  const uint8_t *genome;
  const uint64_t *hash;
  const uint32_t *pos;
  const uint32_t *bucket;
  int shift;
  uint32_t *lo;     // nreads x P: first index of the q-gram's run
  uint32_t *count;  // nreads x P: list length + 1 (its terminating 0)
};

// Bound by the latency of the search's dependent loads: the bucket leaves
// about four of them, where two searches of the whole index took 2 x 23
// (0.36 ms for 200k reads of 100 bp on a 5 Mbp genome).
__global__ void k_lookup(const __grid_constant__ LookupArgs a) {
  const long total = a.nreads * a.S.P;
  const int q = a.S.q;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total;
       t += (long)gridDim.x * blockDim.x) {
    const long r = t / a.S.P;
    const int at = a.S.qpos[t - r * a.S.P];
    const uint8_t *rd = a.reads + r * a.S.m;
    uint64_t h = 1469598103934665603ull;
    for (int i = 0; i < q; ++i) {
      h ^= strand_byte(rd, a.S.m, a.dr, at + i);
      h *= 1099511628211ull;
    }
    uint32_t l = 0, len = 0;
    if (a.bucket) {
      const uint32_t v = (uint32_t)(h >> a.shift);
      const uint32_t end = a.bucket[v + 1];
      l = a.bucket[v];
      uint32_t u = end;
      while (l < u) {  // first index with hash >= h
        const uint32_t mid = l + ((u - l) >> 1);
        if (a.hash[mid] < h) l = mid + 1;
        else u = mid;
      }
      uint32_t e = l;
      u = end;
      while (e < u) {  // first index with hash > h
        const uint32_t mid = e + ((u - e) >> 1);
        if (a.hash[mid] <= h) e = mid + 1;
        else u = mid;
      }
      len = e - l;
    }
    if (len > 0) {  // a hash shared with another q-gram: no list
      const uint8_t *gq = a.genome + a.pos[l];
      for (int i = 0; i < q; ++i)
        if (gq[i] != strand_byte(rd, a.S.m, a.dr, at + i)) {
          len = 0;
          break;
        }
    }
    a.lo[t] = l;
    a.count[t] = len + 1;
  }
}

struct FilterArgs {
  const uint8_t *reads;
  long r0, r1;      // reads of this launch
  long chunk;       // reads per chunk of the reference's data array (its chunk value)
  long nreads;
  int dr;
  FilterShape S;
  const uint8_t *genome;
  long glen;
  const uint32_t *pos;
  const uint32_t *lo, *count;     // per (read, q-gram)
  const long *offs;               // exclusive scan of count
  int32_t *hit_pos;               // (r1 - r0) x kHitsPerRead
  int8_t *hit_flag;
  int32_t *n, *queue;             // per read of the launch
  unsigned long long *made;       // candidates (low half) and perfect hits (high half)
  int *status;
  const int32_t *order;           // the launch's reads (0-based in it), most work first
  uint32_t offset;                // genome position of the chunk's first byte
  int64_t limit;                  // windows end by this genome position
};

// The read's lists on the device: the sorted index's run for each q-gram,
// and the data array's flattened offsets for looks past a list.
struct DevLists {
  const FilterArgs *a;
  long base, c1, cend;
  int P;
  const uint32_t *lo, *cnt;  // this read's lists (shared-memory copies)
  const long *offs;
  uint32_t off;  // the chunk's genome position: values are whole-genome positions
  __device__ uint32_t len(int x) const { return cnt[x] - 1; }
  __device__ uint32_t value(int x, uint32_t i) const { return a->pos[lo[x] + i] + off; }
  __device__ uint32_t at(int x, uint32_t i) const {
    const uint32_t c = cnt[x];
    if (i + 1 < c) return value(x, i);
    if (i + 1 == c) return 0u;
    const long j = offs[x] + (long)i;  // past the list: what follows it
    if (j >= cend) return 0u;
    int y = x + 1;  // in the read's own lists
    while (y < P && offs[y] + (long)cnt[y] <= j) ++y;
    if (y < P) {
      const uint32_t w = (uint32_t)(j - offs[y]);
      return w + 1 < cnt[y] ? value(y, w) : 0u;
    }
    long l = base + P, u = c1 * P - 1;  // or a later read's, by bisection
    while (l < u) {
      const long mid = (l + u + 1) >> 1;
      if (a->offs[mid] <= j) l = mid;
      else u = mid - 1;
    }
    const long w = j - a->offs[l];
    return w + 1 < (long)a->count[l] ? a->pos[a->lo[l] + w] + off : 0u;
  }
  __device__ uint32_t lower(int x, uint32_t from, uint32_t v) const {
    uint32_t l = from, u = cnt[x] - 1;
    while (l < u) {
      const uint32_t mid = (l + u) >> 1;
      if (value(x, mid) < v) l = mid + 1;
      else u = mid;
    }
    return l;
  }
};

constexpr int kFilterWarps = 4;   // warps (reads) per CTA
constexpr int kKeptCache = 96;    // kept positions of a read in shared memory
constexpr int kReadCache = 512;   // bytes of a strand-adjusted read in shared memory

// The positions kept for a read: the first kKeptCache in shared memory, all
// in the read's slice.  Every lane carries the same n, queue and overflow.
struct WarpKept {
  int2 *near_;  // (position, flag) in shared memory
  int32_t *pos;
  int8_t *flag;
  int n, queue, overflow;
  __device__ int2 get(int c) const {
    return c < kKeptCache ? near_[c] : make_int2(pos[c], flag[c]);
  }
  // filter_record (filter_core.cuh) by a whole warp: the kept entries are
  // examined 32 at a time and the first that decides wins, as in the
  // sequential loop; with none deciding, lane 0 appends.
  __device__ void record(int lane, int k, int start, int fl) {
    for (int c0 = 0; c0 < n; c0 += 32) {
      const int c = c0 + lane;
      int code = 0;
      if (c < n) {
        const int2 e = get(c);
        code = kept_decides(e.x, e.y, k, start, fl);
      }
      const unsigned any = __ballot_sync(0xffffffffu, code != 0);
      if (any) {
        if (lane == __ffs(any) - 1 && code == 2) {
          flag[c] = (int8_t)fl;
          if (c < kKeptCache) near_[c].y = fl;
        }
        __syncwarp();
        return;
      }
    }
    if (n >= kHitsPerRead) {
      overflow = 1;
      return;
    }
    if (lane == 0) {
      pos[n] = start;
      flag[n] = (int8_t)fl;
      if (n < kKeptCache) near_[n] = make_int2(start, fl);
    }
    ++n;
    if (start > 0) ++queue;
    __syncwarp();
  }
  // whether an entry kept so far drops a new position (a later change of
  // the entries cannot undo that: they only gain entries and lower flags)
  __device__ bool drops(int k, int start, int fl) const {
    const int cached = n < kKeptCache ? n : kKeptCache;
#pragma unroll 2
    for (int c = 0; c < cached; ++c) {
      const int2 e = near_[c];
      const int d = kept_decides(e.x, e.y, k, start, fl);
      if (d) return d != 2;
    }
    for (int c = cached; c < n; ++c) {
      const int d = kept_decides(pos[c], flag[c], k, start, fl);
      if (d) return d != 2;
    }
    return false;
  }
};

// Whether the genome at `g` spells the read (m bytes).  Reads up to 7 bytes
// past the genome bytes it compares (the buffer has that slack).
__device__ inline bool spells(const uint8_t *g, const uint8_t *read, const uint8_t *cached, int m,
                              int dr) {
  if (m > kReadCache) {
    for (int i = 0; i < m; ++i)
      if (g[i] != strand_byte(read, m, dr, i)) return false;
    return true;
  }
  const uintptr_t ad = (uintptr_t)g;
  const uint32_t *w = reinterpret_cast<const uint32_t *>(ad & ~(uintptr_t)3);
  const uint32_t *c = reinterpret_cast<const uint32_t *>(cached);
  const uint32_t sh = (uint32_t)(ad & 3u) * 8u;
  uint32_t lo = w[0];
  for (int i = 0; i < m; i += 4) {
    const uint32_t hi = *++w;
    uint32_t d = __funnelshift_r(lo, hi, sh) ^ *c++;
    if (m - i < 4) d &= (1u << (8 * (m - i))) - 1u;
    if (d) return false;
    lo = hi;
  }
  return true;
}

// One warp per read.  The positions of the first-half q-grams, in the
// reference's order (q-grams ascending, list order), are taken 32 at a time,
// a lane each: its perfect match and the pair that brings its count to the
// threshold (position_hit), dropped at once where a kept entry drops them;
// what is left is recorded one after the other.  Warps take the launch's
// reads in the order `order` gives (most estimated work first), so long
// reads start early and short ones fill in.
//
// Bound by the latency of the searches' loads (L1 and L2 hold the lists).  A
// lane per pair item and error zone instead, one position at a time, took
// 9.1k warp instructions and 15 ns a read of 100 bp on the repeat-rich 5 Mbp
// genome.
__global__ void __launch_bounds__(32 * kFilterWarps) k_filter(const __grid_constant__ FilterArgs fa) {
  __shared__ uint32_t s_lo[kFilterWarps][kFilterMaxQgrams], s_cnt[kFilterWarps][kFilterMaxQgrams];
  __shared__ long s_offs[kFilterWarps][kFilterMaxQgrams];
  __shared__ uint32_t s_first[kFilterWarps][kFilterMaxQgrams / 2 + 1];
  __shared__ int2 s_kept[kFilterWarps][kKeptCache];
  __shared__ __align__(4) uint8_t s_read[kFilterWarps][kReadCache];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long wi = blockIdx.x * (long)kFilterWarps + w;
  if (wi >= fa.r1 - fa.r0) return;  // the whole warp
  const long lr = fa.order[wi];
  const long r = fa.r0 + lr;
  const FilterShape &S = fa.S;
  const int P = S.P, k = S.k, half = S.half, q = S.q, m = S.m, dr = fa.dr;
  const long c1 = min((r / fa.chunk + 1) * fa.chunk, fa.nreads);
  for (int x = lane; x < P; x += 32) {
    s_lo[w][x] = fa.lo[r * P + x];
    s_cnt[w][x] = fa.count[r * P + x];
    s_offs[w][x] = fa.offs[r * P + x];
  }
  __syncwarp();
  const DevLists L{&fa,     r * P,   c1,        fa.offs[c1 * P - 1] + (long)fa.count[c1 * P - 1],
                   P,       s_lo[w], s_cnt[w],  s_offs[w],
                   fa.offset};
  const int goff = (int)fa.offset;
  const uint8_t *rd = fa.reads + r * m;
  WarpKept h{s_kept[w], fa.hit_pos + lr * kHitsPerRead, fa.hit_flag + lr * kHitsPerRead, 0, 0, 0};
  // positions of the first-half lists back to back (a list that begins with
  // a 0 reads as empty)
  uint32_t total = 0;
  for (int a = 0; a < half; ++a) {
    if (lane == 0) s_first[w][a] = total;
    const uint32_t n = L.len(a);
    if (n > 0 && L.value(a, 0) != 0) total += n;
  }
  if (lane == 0) s_first[w][half] = total;
  if (total > 0 && m <= kReadCache)
    for (int i = lane; i < m; i += 32) s_read[w][i] = strand_byte(rd, m, dr, i);
  __syncwarp();
  for (uint32_t t0 = 0; t0 < total; t0 += 32) {
    const uint32_t t = t0 + lane;
    bool perfect = false, hit = false;
    int g1 = 0, flag = 0, start = 0;
    if (t < total) {
      int a = 0;
      while (s_first[w][a + 1] <= t) ++a;
      const uint32_t off = t - s_first[w][a];
      const uint32_t pa = L.value(a, off);
      g1 = (int)(pa - ((uint32_t)a * q + 1)) + 1;
      if (g1 - goff > 0) {  // a start after the chunk's first byte
        const long l1 = (long)g1 - goff;
        perfect = l1 + m <= fa.glen && spells(fa.genome + l1, rd, s_read[w], m, dr) &&
                  !h.drops(k, -g1, 0);
        hit = position_hit(S, dr, L, a, off, pa, flag, start) && !h.drops(k, start, flag);
      }
    }
    for (unsigned left = __ballot_sync(0xffffffffu, perfect || hit); left; left &= left - 1) {
      const int src = __ffs(left) - 1;
      if (__shfl_sync(0xffffffffu, perfect, src))
        h.record(lane, k, -__shfl_sync(0xffffffffu, g1, src), 0);
      if (__shfl_sync(0xffffffffu, hit, src))
        h.record(lane, k, __shfl_sync(0xffffffffu, start, src),
                 __shfl_sync(0xffffffffu, flag, src));
    }
  }
  // how many of the kept positions are candidates (their windows fit the
  // genome) and perfect hits
  int cand = 0, exact = 0;
  for (int c = lane; c < h.n; c += 32) {
    const int2 e = h.get(c);
    int so, eo;
    flank_of(e.y, k, so, eo);
    cand += e.x > 0 && (int64_t)e.x + m + so + eo <= fa.limit;
    exact += e.y == 0;
  }
  cand = __reduce_add_sync(0xffffffffu, cand);
  exact = __reduce_add_sync(0xffffffffu, exact);
  if (lane == 0) {
    fa.n[lr] = h.n;
    fa.queue[lr] = h.queue;
    fa.made[lr] = (unsigned long long)(unsigned)cand | (unsigned long long)(unsigned)exact << 32;
    if (h.overflow) atomicOr(fa.status, 1);
  }
}

// A read's estimated filter work: the positions of its first-half q-grams.
__global__ void k_work(const uint32_t *count, long r0, long cnt, FilterShape S, uint32_t *key,
                       int32_t *idx) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < cnt;
       i += (long)gridDim.x * blockDim.x) {
    const long r = r0 + i;
    unsigned long long w = 0;
    for (int a = 0; a < S.half; ++a) w += count[r * S.P + a] - 1;
    key[i] = (uint32_t)(w < 0xffffffffull ? w : 0xffffffffull);
    idx[i] = (int32_t)i;
  }
}

// A launch's candidates and perfect hits back to back, in read order and
// the order the filter kept them; at: exclusive scan of `made`.  A warp per
// read.
struct CallArgs {
  const int32_t *hit_pos;
  const int8_t *hit_flag;
  const int32_t *n;
  const unsigned long long *at;
  long nr;
  int32_t r0;
  int m, k;
  int64_t limit;
  int32_t *ids, *pos, *perfect_ids, *perfect_pos;
  int8_t *dirs;
};

__global__ void __launch_bounds__(256) k_calls(const __grid_constant__ CallArgs a) {
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * (blockDim.x >> 5);
  for (long r = blockIdx.x * (long)(blockDim.x >> 5) + (threadIdx.x >> 5); r < a.nr; r += warps) {
    const int n = a.n[r];
    uint32_t c = (uint32_t)a.at[r], p = (uint32_t)(a.at[r] >> 32);
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      int pos = 0, flag = 0, so = 0, eo = 0;
      if (i < n) {
        pos = a.hit_pos[r * kHitsPerRead + i];
        flag = a.hit_flag[r * kHitsPerRead + i];
      }
      flank_of(flag, a.k, so, eo);
      const bool cand = i < n && pos > 0 && (int64_t)pos + a.m + so + eo <= a.limit;
      const bool exact = i < n && flag == 0;
      const unsigned bc = __ballot_sync(0xffffffffu, cand), bp = __ballot_sync(0xffffffffu, exact);
      const unsigned below = (1u << lane) - 1u;
      if (cand) {
        const uint32_t t = c + __popc(bc & below);
        a.ids[t] = a.r0 + (int32_t)r;
        a.pos[t] = pos;
        a.dirs[t] = (int8_t)flag;
      }
      if (exact) {
        const uint32_t t = p + __popc(bp & below);
        a.perfect_ids[t] = a.r0 + (int32_t)r;
        a.perfect_pos[t] = -pos;
      }
      c += __popc(bc);
      p += __popc(bp);
    }
  }
}

// Device memory that grows, stream-ordered on the filter's stream: a
// growth neither waits for the device's other work (a plain cudaFree
// synchronizes the whole device, so one filter's growth stalled the
// aligner and the other filters of a server) nor for the host.  `slack`
// extra elements are taken on a growth, for buffers sized by the request.
template <typename T>
struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  cudaError_t ensure(size_t count, cudaStream_t s, size_t slack = 0) {
    if (count <= n) return cudaSuccess;
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
    n = 0;
    const size_t want = count + slack;
    const cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&p), want * sizeof(T) + 64, s);
    if (e == cudaSuccess) n = want;
    else p = nullptr;
    return e;
  }
  void release(cudaStream_t s) {
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
    n = 0;
  }
};

// Pinned host memory that grows: copies back from the device into it run
// at full speed and without staging.
template <typename T>
struct HBuf {
  T *p = nullptr;
  size_t n = 0;
  cudaError_t ensure(size_t count) {
    if (count <= n) return cudaSuccess;
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
    const size_t want = std::max(count + count / 2, 2 * n) + 64;
    const cudaError_t e = cudaMallocHost(&p, want * sizeof(T));
    if (e == cudaSuccess) n = want;
    return e;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
  }
};

// Host memory that grows (uninitialised; contents kept on a growth).
template <typename T>
struct GrowBuf {
  T *p = nullptr;
  size_t n = 0, cap = 0;
  bool grow(size_t count) {  // to n = count
    if (count > cap || !p) {
      const size_t want = std::max(count + count / 2, (size_t)1024);
      void *q = realloc(p, want * sizeof(T));
      if (!q) return false;
      p = static_cast<T *>(q);
      cap = want;
    }
    n = count;
    return true;
  }
  ~GrowBuf() { free(p); }
};

// A launch's results on their way to the host: one block of device memory,
// one of pinned memory and one copy for its candidates and perfect hits.
struct LaunchOut {
  DBuf<uint8_t> dev;
  HBuf<uint8_t> host;
  HBuf<unsigned long long> counts;  // places by read, the totals, the queue counts
  cudaEvent_t filtered = nullptr, copied = nullptr, placed = nullptr;
};

// Where a launch's nc candidates and np perfect hits lie in its block.
struct OutBlock {
  size_t ids, pos, perfect_ids, perfect_pos, dirs, bytes;
  OutBlock(size_t nc, size_t np)
      : ids(0), pos(4 * nc), perfect_ids(8 * nc), perfect_pos(8 * nc + 4 * np),
        dirs(8 * nc + 8 * np), bytes(9 * nc + 8 * np) {}
};

}  // namespace

struct saru_filter {
  int device = 0, m = 0, k = 0;
  FilterShape S{};
  long glen = 0, nidx = 0;
  int64_t offset = 0, limit = -1;  // the chunk's genome position; windows end by limit
  cudaStream_t s = nullptr;
  DBuf<uint8_t> genome, reads, temp;
  DBuf<uint64_t> hash, hash_s;
  DBuf<uint32_t> pos, pos_s;
  DBuf<long> offs;
  DBuf<uint32_t> lo, count, bucket;
  DBuf<unsigned long long> made, at;
  DBuf<int32_t> hit_pos, n, queue, widx;
  DBuf<uint32_t> wkey;
  DBuf<int8_t> hit_flag;
  DBuf<int> status;
  int bucket_shift = 0;
  cudaStream_t s_out = nullptr;  // copies of results out
  LaunchOut out[2];              // one launch's results are copied out while the next runs
  // the last run's calls (filter_calls.h), storage kept across runs
  std::vector<int64_t> call_begin;
  GrowBuf<int32_t> c_ids, c_pos, p_ids, p_pos;
  GrowBuf<int8_t> c_dirs;
  float last_ms = 0.f;
};

namespace {

int fail(const char *what, cudaError_t e) {
  std::string msg = std::string(what) + ": " + cudaGetErrorString(e);
  saru::set_last_error(msg.c_str());
  return SARU_E_CUDA;
}

}  // namespace

extern "C" {

saru_filter *saru_filter_create(const char *genome, int64_t genome_len, int32_t read_length,
                                int32_t k, int32_t device) {
  saru::set_last_error("");
  if (device < 0 && cudaGetDevice(&device) != cudaSuccess) device = 0;  // the current one
  auto *f = new saru_filter();
  f->device = device;
  f->m = read_length;
  f->k = k;
  f->glen = genome_len;
  if (!genome || genome_len < 1 || read_length < 2 || k < 0 ||
      !filter_shape(read_length, k, &f->S) || f->S.q > 4 * kFilterMaxQgrams) {
    saru::set_last_error("saru_filter_create: a genome, read_length >= 2, k >= 0 and a q-gram "
                         "layout of at most 64 q-grams");
    delete f;
    return nullptr;
  }
  const int q = f->S.q;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&f->s, cudaStreamNonBlocking);
  f->nidx = genome_len >= q ? genome_len - q + 1 : 0;
  const long n = f->nidx;
  if (e == cudaSuccess) e = f->genome.ensure((size_t)genome_len, f->s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(f->genome.p, genome, (size_t)genome_len, cudaMemcpyHostToDevice, f->s);
  if (e == cudaSuccess && n > 0) {
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint64_t *)nullptr, (uint64_t *)nullptr,
                                    (uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0, 64,
                                    f->s);
    if ((e = f->hash.ensure(n, f->s)) == cudaSuccess &&
        (e = f->hash_s.ensure(n, f->s)) == cudaSuccess &&
        (e = f->pos.ensure(n, f->s)) == cudaSuccess &&
        (e = f->pos_s.ensure(n, f->s)) == cudaSuccess &&
        (e = f->temp.ensure(tb, f->s)) == cudaSuccess &&
        (e = f->status.ensure(1, f->s)) == cudaSuccess) {
      k_qgram_hash<<<1184, 256, 0, f->s>>>(f->genome.p, n, q, f->hash.p, f->pos.p);
      e = cudaGetLastError();
      if (e == cudaSuccess)
        e = cub::DeviceRadixSort::SortPairs(f->temp.p, tb, f->hash.p, f->hash_s.p, f->pos.p,
                                            f->pos_s.p, (int)n, 0, 64, f->s);
      if (e == cudaSuccess) e = cudaMemsetAsync(f->status.p, 0, sizeof(int), f->s);
      if (e == cudaSuccess) {
        k_index_check<<<1184, 256, 0, f->s>>>(f->hash_s.p, f->pos_s.p, n, f->genome.p, q,
                                              f->status.p);
        e = cudaGetLastError();
      }
      int flag = 0;
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(&flag, f->status.p, sizeof(int), cudaMemcpyDeviceToHost, f->s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(f->s);
      if (e == cudaSuccess && flag) {
        saru::set_last_error("saru_filter_create: two different q-grams share a 64-bit hash");
        saru_filter_destroy(f);
        return nullptr;
      }
      f->hash.release(f->s);
      f->pos.release(f->s);
      // about ten hashes a bucket
      int bits = 4;
      while (bits < 24 && (16l << bits) < n) ++bits;
      f->bucket_shift = 64 - bits;
      if (e == cudaSuccess) e = f->bucket.ensure(((size_t)1 << bits) + 1, f->s);
      if (e == cudaSuccess) {
        k_buckets<<<1184, 256, 0, f->s>>>(f->hash_s.p, n, f->bucket_shift, 1u << bits,
                                          f->bucket.p);
        e = cudaGetLastError();
      }
    }
  }
  // the genome (saru_filter_genome) is usable on any stream once this returns
  if (e == cudaSuccess) e = cudaStreamSynchronize(f->s);
  if (e != cudaSuccess) {
    fail("saru_filter_create", e);
    saru_filter_destroy(f);
    return nullptr;
  }
  saru::count_launch();
  return f;
}

int saru_filter_run(saru_filter *f, const char *reads, int32_t nreads, int32_t do_reverse,
                    uint32_t chunk_value, int64_t *counts) {
  saru::set_last_error("");
  if (!f || !counts || nreads < 0 || (nreads > 0 && !reads) || chunk_value < 1 ||
      (do_reverse != 0 && do_reverse != 4)) {
    saru::set_last_error("saru_filter_run: reads, chunk_value >= 1, do_reverse 0 or 4");
    return SARU_E_INVALID;
  }
  const long read_chunk = (long)chunk_value;  // the data array's chunk of reads
  cudaSetDevice(f->device);
  const FilterShape &S = f->S;
  const long nr = nreads, P = S.P, m = f->m;
  const int64_t limit = f->limit >= 0 ? f->limit : f->glen;
  f->call_begin.assign(1, 0);
  f->c_ids.n = f->c_pos.n = f->c_dirs.n = f->p_ids.n = f->p_pos.n = 0;
  uint32_t queued = 0;
  // a call's end (filter_calls.h, close_call)
  auto close_call = [&](int64_t end) {
    if (end > f->call_begin.back()) f->call_begin.push_back(end);
    queued = 0;
  };
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaError_t e = cudaSuccess;
  int rc = SARU_OK;
  float ms = 0.f;
  if (nr > 0) {
    const long lists = nr * P;
    size_t tb = 0;
    cub::DeviceScan::ExclusiveScan(nullptr, tb, (uint32_t *)nullptr, (long *)nullptr, AddLong{},
                                   0L, (int)lists, f->s);
    size_t tb2 = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb2, (unsigned long long *)nullptr,
                                  (unsigned long long *)nullptr, (int)kReadsPerLaunch + 1, f->s);
    size_t tb3 = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, tb3, (uint32_t *)nullptr,
                                              (uint32_t *)nullptr, (int32_t *)nullptr,
                                              (int32_t *)nullptr, (int)kReadsPerLaunch, 0, 32,
                                              f->s);
    const long batch = std::min<long>(nr, kReadsPerLaunch);
    // buffers sized by the request's reads take half again on a growth;
    // those sized by a launch stop growing at kReadsPerLaunch reads
    cudaStream_t s = f->s;
    // (a server builds filters that a worker may never run)
    if (!f->s_out) e = cudaStreamCreateWithFlags(&f->s_out, cudaStreamNonBlocking);
    for (LaunchOut &o : f->out)
      for (cudaEvent_t *ev : {&o.filtered, &o.copied, &o.placed})
        if (e == cudaSuccess && !*ev) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e != cudaSuccess ||
        (e = f->reads.ensure((size_t)(nr * m), s, (size_t)(nr * m) / 2)) != cudaSuccess ||
        (e = f->lo.ensure(lists, s, lists / 2)) != cudaSuccess ||
        (e = f->count.ensure(lists, s, lists / 2)) != cudaSuccess ||
        (e = f->offs.ensure(lists, s, lists / 2)) != cudaSuccess ||
        (e = f->temp.ensure(std::max(std::max(tb, tb2), tb3), s)) != cudaSuccess ||
        (e = f->wkey.ensure((size_t)batch * 2, s)) != cudaSuccess ||
        (e = f->widx.ensure((size_t)batch * 2, s)) != cudaSuccess ||
        (e = f->hit_pos.ensure((size_t)batch * kHitsPerRead, s)) != cudaSuccess ||
        (e = f->hit_flag.ensure((size_t)batch * kHitsPerRead, s)) != cudaSuccess ||
        (e = f->n.ensure(batch, s)) != cudaSuccess || (e = f->queue.ensure(batch, s)) != cudaSuccess ||
        (e = f->made.ensure(batch + 1, s)) != cudaSuccess ||
        (e = f->at.ensure(batch + 1, s)) != cudaSuccess ||
        (e = f->status.ensure(1, s)) != cudaSuccess) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return fail("saru_filter_run", e);
    }
    cudaEventRecord(e0, s);
    e = cudaMemcpyAsync(f->reads.p, reads, (size_t)(nr * m), cudaMemcpyHostToDevice, s);
    LookupArgs la{f->reads.p, nr, do_reverse, S, f->genome.p, f->hash_s.p, f->pos_s.p,
                  f->bucket.p, f->bucket_shift, f->lo.p, f->count.p};
    if (e == cudaSuccess) {
      k_lookup<<<(unsigned)std::min<long>((lists + 255) / 256, 65535), 256, 0, s>>>(la);
      e = cudaGetLastError();
    }
    // one scan over all reads: each chunk's lists stay contiguous, and the
    // filter bounds its look past a list by its chunk's end
    if (e == cudaSuccess)
      e = cub::DeviceScan::ExclusiveScan(f->temp.p, tb, f->count.p, f->offs.p, AddLong{}, 0L,
                                         (int)lists, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(f->status.p, 0, sizeof(int), s);
    // filters the reads of launch li (from r0) and sends their counts home
    auto filter_launch = [&](long r0, LaunchOut &o) -> cudaError_t {
      const long r1 = std::min(nr, r0 + batch), cnt = r1 - r0;
      cudaError_t x;
      k_work<<<(unsigned)((cnt + 255) / 256), 256, 0, s>>>(f->count.p, r0, cnt, S, f->wkey.p,
                                                           f->widx.p);
      if ((x = cudaGetLastError()) != cudaSuccess ||
          (x = cub::DeviceRadixSort::SortPairsDescending(
               f->temp.p, tb3, f->wkey.p, f->wkey.p + batch, f->widx.p, f->widx.p + batch,
               (int)cnt, 0, 32, s)) != cudaSuccess)
        return x;
      FilterArgs fa{f->reads.p, r0, r1, read_chunk, nr, do_reverse, S, f->genome.p,
                    f->glen, f->pos_s.p, f->lo.p, f->count.p, f->offs.p, f->hit_pos.p,
                    f->hit_flag.p, f->n.p, f->queue.p, f->made.p, f->status.p,
                    f->widx.p + batch, (uint32_t)f->offset, limit};
      k_filter<<<(unsigned)((cnt + kFilterWarps - 1) / kFilterWarps), 32 * kFilterWarps, 0, s>>>(
          fa);
      if ((x = cudaGetLastError()) != cudaSuccess ||
          // (the sum's last output, the totals, does not read the last input)
          (x = cub::DeviceScan::ExclusiveSum(f->temp.p, tb2, f->made.p, f->at.p, (int)cnt + 1,
                                             s)) != cudaSuccess ||
          (x = o.counts.ensure((size_t)batch + 1 + (size_t)batch / 2 + 1)) != cudaSuccess ||
          (x = cudaMemcpyAsync(o.counts.p, f->at.p, 8 * ((size_t)cnt + 1), cudaMemcpyDeviceToHost,
                               s)) != cudaSuccess ||
          (x = cudaMemcpyAsync(o.counts.p + cnt + 1, f->queue.p, 4 * (size_t)cnt,
                               cudaMemcpyDeviceToHost, s)) != cudaSuccess)
        return x;
      saru::count_launch();
      return cudaEventRecord(o.filtered, s);
    };
    // its candidates and perfect hits to the host (s_out), once the counts
    // are there
    auto calls_launch = [&](long r0, LaunchOut &o) -> cudaError_t {
      const long cnt = std::min(nr, r0 + batch) - r0;
      cudaError_t x = cudaEventSynchronize(o.filtered);
      if (x != cudaSuccess) return x;
      const size_t nc = (uint32_t)o.counts.p[cnt], np = (size_t)(o.counts.p[cnt] >> 32);
      const OutBlock at(nc, np);
      if ((x = o.dev.ensure(at.bytes + 1, s, at.bytes / 2)) != cudaSuccess ||
          (x = o.host.ensure(at.bytes + 1)) != cudaSuccess)
        return x;
      auto ints = [&](size_t off) { return reinterpret_cast<int32_t *>(o.dev.p + off); };
      CallArgs ca{f->hit_pos.p, f->hit_flag.p, f->n.p, f->at.p, cnt, (int32_t)r0, f->m, f->k,
                  limit, ints(at.ids), ints(at.pos), ints(at.perfect_ids), ints(at.perfect_pos),
                  reinterpret_cast<int8_t *>(o.dev.p + at.dirs)};
      k_calls<<<(unsigned)std::min<long>((cnt + 7) / 8, 148 * 8), 256, 0, s>>>(ca);
      if ((x = cudaGetLastError()) != cudaSuccess ||
          (x = cudaEventRecord(o.placed, s)) != cudaSuccess ||
          (x = cudaStreamWaitEvent(f->s_out, o.placed, 0)) != cudaSuccess)
        return x;
      if (at.bytes && (x = cudaMemcpyAsync(o.host.p, o.dev.p, at.bytes, cudaMemcpyDeviceToHost,
                                           f->s_out)) != cudaSuccess)
        return x;
      return cudaEventRecord(o.copied, f->s_out);
    };
    // appended to the run's calls, call boundaries set
    auto take_launch = [&](long r0, LaunchOut &o) -> cudaError_t {
      const long cnt = std::min(nr, r0 + batch) - r0;
      const cudaError_t x = cudaEventSynchronize(o.copied);
      if (x != cudaSuccess) return x;
      const size_t nc = (uint32_t)o.counts.p[cnt], np = (size_t)(o.counts.p[cnt] >> 32);
      const size_t c0 = f->c_ids.n, p0 = f->p_ids.n;
      const OutBlock at(nc, np);
      if (!f->c_ids.grow(c0 + nc) || !f->c_pos.grow(c0 + nc) || !f->c_dirs.grow(c0 + nc) ||
          !f->p_ids.grow(p0 + np) || !f->p_pos.grow(p0 + np))
        return cudaErrorMemoryAllocation;
      memcpy(f->c_ids.p + c0, o.host.p + at.ids, 4 * nc);
      memcpy(f->c_pos.p + c0, o.host.p + at.pos, 4 * nc);
      memcpy(f->c_dirs.p + c0, o.host.p + at.dirs, nc);
      memcpy(f->p_ids.p + p0, o.host.p + at.perfect_ids, 4 * np);
      memcpy(f->p_pos.p + p0, o.host.p + at.perfect_pos, 4 * np);
      const int32_t *queue = reinterpret_cast<const int32_t *>(o.counts.p + cnt + 1);
      for (long i = 0; i < cnt; ++i) {
        queued += (uint32_t)queue[i];
        if (queued > chunk_value) close_call((int64_t)(c0 + (uint32_t)o.counts.p[i + 1]));
      }
      return cudaSuccess;
    };
    long r0 = 0;
    int set = 0;
    if (e == cudaSuccess) e = filter_launch(0, f->out[0]);
    for (; r0 < nr && e == cudaSuccess; r0 += batch, set ^= 1) {
      e = calls_launch(r0, f->out[set]);
      // the next launch runs while this one's results are copied and taken
      if (e == cudaSuccess && r0 + batch < nr) e = filter_launch(r0 + batch, f->out[set ^ 1]);
      if (e == cudaSuccess) e = take_launch(r0, f->out[set]);
    }
    int flag = 0;
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&flag, f->status.p, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaEventRecord(e1, s);
    // nothing of this run is in flight when it returns, errors included
    const cudaError_t es = cudaStreamSynchronize(s), eo = cudaStreamSynchronize(f->s_out);
    if (e == cudaSuccess) e = es != cudaSuccess ? es : eo;
    if (e != cudaSuccess) rc = fail("saru_filter_run", e);
    else if (flag) {
      saru::set_last_error("saru_filter_run: a read kept more positions than the filter holds");
      rc = SARU_E_OVERFLOW;
    }
    if (rc == SARU_OK) cudaEventElapsedTime(&ms, e0, e1);
  }
  // the last call: only when positions are queued (else the candidates since
  // the last call are never submitted, as in the reference)
  if (queued > 0) close_call((int64_t)f->c_ids.n);
  else f->c_ids.n = f->c_pos.n = f->c_dirs.n = (size_t)f->call_begin.back();
  f->last_ms = ms;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  counts[0] = (int64_t)f->call_begin.size() - 1;
  counts[1] = (int64_t)f->c_ids.n;
  counts[2] = (int64_t)f->p_ids.n;
  return rc;
}

int saru_filter_results(const saru_filter *f, int64_t *call_begin, int32_t *ids, int32_t *pos,
                        int8_t *dirs, int32_t *perfect_ids, int32_t *perfect_pos) {
  if (!f) return SARU_E_INVALID;
  const auto copy = [](void *to, const void *from, size_t bytes) {
    if (to && bytes) memcpy(to, from, bytes);
  };
  copy(call_begin, f->call_begin.data(), f->call_begin.size() * 8);
  copy(ids, f->c_ids.p, f->c_ids.n * 4);
  copy(pos, f->c_pos.p, f->c_pos.n * 4);
  copy(dirs, f->c_dirs.p, f->c_dirs.n);
  copy(perfect_ids, f->p_ids.p, f->p_ids.n * 4);
  copy(perfect_pos, f->p_pos.p, f->p_pos.n * 4);
  return SARU_OK;
}

double saru_filter_last_ms(const saru_filter *f) { return f ? f->last_ms : -1.0; }

const char *saru_filter_genome(const saru_filter *f) {
  return f ? reinterpret_cast<const char *>(f->genome.p) : nullptr;
}

int saru_filter_set_chunk(saru_filter *f, int64_t offset, int64_t limit) {
  saru::set_last_error("");
  if (!f || offset < 0 || limit < offset || offset + f->glen > (int64_t)UINT32_MAX) {
    saru::set_last_error("saru_filter_set_chunk: offset >= 0, limit >= offset, positions in 32 bits");
    return SARU_E_INVALID;
  }
  f->offset = offset;
  f->limit = limit;
  return SARU_OK;
}

void saru_filter_destroy(saru_filter *f) {
  if (!f) return;
  int caller_dev = 0;  // the caller's current device, restored before returning
  const bool had_dev = cudaGetDevice(&caller_dev) == cudaSuccess;
  cudaSetDevice(f->device);
  if (f->s) cudaStreamSynchronize(f->s);
  if (f->s_out) cudaStreamSynchronize(f->s_out);
  f->genome.release(f->s);
  f->reads.release(f->s);
  f->temp.release(f->s);
  f->hash.release(f->s);
  f->hash_s.release(f->s);
  f->pos.release(f->s);
  f->pos_s.release(f->s);
  f->bucket.release(f->s);
  f->lo.release(f->s);
  f->count.release(f->s);
  f->offs.release(f->s);
  f->made.release(f->s);
  f->at.release(f->s);
  f->hit_pos.release(f->s);
  f->hit_flag.release(f->s);
  f->n.release(f->s);
  f->queue.release(f->s);
  f->status.release(f->s);
  f->wkey.release(f->s);
  f->widx.release(f->s);
  for (LaunchOut &o : f->out) {
    o.dev.release(f->s);
    o.host.release();
    o.counts.release();
    for (cudaEvent_t ev : {o.filtered, o.copied, o.placed})
      if (ev) cudaEventDestroy(ev);
  }
  if (f->s_out) cudaStreamDestroy(f->s_out);
  if (f->s) {
    cudaStreamSynchronize(f->s);  // the stream-ordered frees
    cudaStreamDestroy(f->s);
  }
  delete f;
  if (had_dev) cudaSetDevice(caller_dev);
}

}  // extern "C"
