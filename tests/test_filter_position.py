"""The filter position by position (filter_core.cuh: position_hit and
kept_decides, what the device kernel runs a lane per position) keeps exactly
what the step-by-step restatement (filter_read) keeps, over the reference's
literal data array: repeat-rich and low-complexity genomes, empty lists that
run into the next ones, q-grams at genome position 0, genome chunks, read
lengths and error counts whose threshold is 1 or more.  CPU only."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SRC = r'''
#include <stdio.h>
#include <string.h>
#include <string>
#include <unordered_map>
#include <vector>
#include "filter_core.cuh"
using namespace saru;
static uint64_t st;
static uint32_t rnd(uint32_t n) {
  st = st * 6364136223846793005ull + 1442695040888963407ull;
  return (uint32_t)(st >> 33) % n;
}
struct Lists {
  const std::vector<uint32_t> *data;
  const size_t *offs, *lens;
  uint32_t len(int x) const { return (uint32_t)lens[x]; }
  uint32_t at(int x, uint32_t i) const {
    const size_t j = offs[x] + i;
    return j < data->size() ? (*data)[j] : 0u;
  }
  uint32_t value(int x, uint32_t i) const { return (*data)[offs[x] + i]; }
  int find(int x, uint32_t lo, uint32_t want) const {
    for (uint32_t i = lo; i < lens[x]; ++i)
      if ((*data)[offs[x] + i] == want) return (int)i;
    return -1;
  }
  uint32_t lower(int x, uint32_t from, uint32_t v) const {
    uint32_t i = from;
    while (i < lens[x] && (*data)[offs[x] + i] < v) ++i;
    return i;
  }
};
struct Event { int start, flag; bool any; };
int main(int argc, char **argv) {
  int m, k, unit, offset;
  unsigned seed;
  sscanf(argv[1], "%d,%d,%d,%d,%u", &m, &k, &unit, &offset, &seed);
  st = seed * 77777u + 5;
  FilterShape S;
  if (!filter_shape(m, k, &S)) return 2;
  const int glen = 6000, nreads = 60;
  std::string g;
  std::string motif;
  for (int i = 0; i < unit; ++i) motif += "ACGT"[rnd(4)];
  while ((int)g.size() < glen) {
    if (rnd(2)) { std::string c = motif; if (rnd(2)) c[rnd(unit)] = "ACGTN"[rnd(5)]; g += c; }
    else for (int i = 0; i < unit; ++i) g += "ACGT"[rnd(4)];
  }
  g.resize(glen);
  std::unordered_map<std::string, std::vector<uint32_t>> index;
  for (int p = 0; p + S.q <= glen; ++p) index[g.substr(p, S.q)].push_back(p + offset);
  std::vector<uint32_t> data;
  std::vector<size_t> offs, lens;
  std::vector<std::string> reads;
  for (int r = 0; r < nreads; ++r) {
    std::string rd = g.substr(r ? rnd(glen - m - 1) : 0, m + 1);
    for (int e = rnd(2 * k + 2); e > 0; --e) {
      const int at = rnd(m);
      if (rnd(3)) rd[at] = "ACGTN"[rnd(5)];
      else { rd.erase(at, 1); rd += 'A'; }
    }
    rd.resize(m);
    reads.push_back(rd);
    for (int x = 0; x < S.P; ++x) {
      offs.push_back(data.size());
      auto it = index.find(rd.substr(S.qpos[x], S.q));
      const bool has = it != index.end() && rnd(12);  // now and then a list goes missing
      if (has) data.insert(data.end(), it->second.begin(), it->second.end());
      lens.push_back(has ? it->second.size() : 0);
      data.push_back(0);
    }
  }
  const int cap = 4096;
  std::vector<int32_t> p1(cap), p2(cap);
  std::vector<int8_t> f1(cap), f2(cap);
  long kept = 0;
  for (int r = 0; r < nreads; ++r)
    for (int dr = 0; dr <= 4; dr += 4) {
      Lists L{&data, &offs[r * S.P], &lens[r * S.P]};
      auto perfect = [&](int g1) {
        const long l1 = (long)g1 - offset;
        return l1 + m <= glen && memcmp(g.data() + l1, reads[r].data(), m) == 0;
      };
      ReadHits a{p1.data(), f1.data(), cap, 0, 0, 0}, b{p2.data(), f2.data(), cap, 0, 0, 0};
      filter_read(S, dr, L, perfect, a, offset);
      std::vector<std::pair<int, uint32_t>> flat;
      for (int x = 0; x < S.half; ++x)
        if (L.len(x) && L.at(x, 0))
          for (uint32_t o = 0; o < L.len(x); ++o) flat.push_back({x, o});
      for (size_t t0 = 0; t0 < flat.size(); t0 += 32) {  // a warp's positions at once
        Event ev[32][2];
        const size_t n = std::min<size_t>(32, flat.size() - t0);
        for (size_t i = 0; i < n; ++i) {
          const int x = flat[t0 + i].first;
          const uint32_t pa = L.at(x, flat[t0 + i].second);
          const int gs = (int)(pa - ((uint32_t)x * S.q + 1));
          ev[i][0].any = ev[i][1].any = false;
          if (gs + 1 - offset <= 0) continue;
          ev[i][0] = Event{-(gs + 1), 0, perfect(gs + 1)};
          ev[i][1].any = position_hit(S, dr, L, x, flat[t0 + i].second, pa, ev[i][1].flag,
                                      ev[i][1].start);
          for (auto &e : ev[i])  // what the entries kept so far already drop
            for (int c = 0; e.any && c < b.n; ++c) {
              const int d = kept_decides(b.pos[c], b.flag[c], k, e.start, e.flag);
              if (d == 2) break;
              if (d) e.any = false;
            }
        }
        for (size_t i = 0; i < n; ++i)
          for (auto &e : ev[i])
            if (e.any) filter_record(b, k, S.tresh, e.start, e.flag, S.tresh);
      }
      kept += a.n;
      if (a.n != b.n || a.queue != b.queue || memcmp(a.pos, b.pos, 4 * a.n) ||
          memcmp(a.flag, b.flag, a.n)) {
        printf("read %d dr %d: %d kept, %d by position\n", r, dr, a.n, b.n);
        return 1;
      }
    }
  printf("same %ld\n", kept);
  return 0;
}
'''

CASES = [(36, 2), (36, 3), (100, 5), (30, 4), (24, 5), (50, 1), (64, 0), (150, 9)]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("fpos")
    (d / "f.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "saruman_b200" / "csrc"),
                    str(d / "f.cpp"), "-o", str(d / "f")], check=True)
    return d / "f"


@pytest.mark.parametrize("m,k", CASES)
def test_positions_keep_what_the_filter_keeps(exe, m, k):
    kept = 0
    for unit in (13, 40, 300):
        for offset in (0, 5000):
            for seed in range(4):
                r = subprocess.run([str(exe), f"{m},{k},{unit},{offset},{seed}"],
                                   capture_output=True, text=True)
                assert r.returncode == 0, r.stdout
                kept += int(r.stdout.split()[1])
    assert kept > 1000
