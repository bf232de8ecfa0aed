"""Host planners of the FP64 contractions (plan_direct, complex_map, f64tc::plan_group) on the CPU: their
tables, walked in integers as the kernels walk them, give what fusing the operands, multiplying and
splitting the result give, every element written once; output tiles, their pieces along K, packing
items and counts cover each sector GEMM once, in both orientations."""
import os
import shutil
import subprocess

import pytest

import mps_gb300.build as build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mps_gb300", "csrc")
CUDA = os.path.dirname(os.path.dirname(build.nvcc())) if shutil.which("g++") else ""

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <map>
#include <random>
#include <set>
#include "copy_decode.hpp"
#include "direct.hpp"
using namespace mpsg;
typedef std::vector<int64_t> Vec;

#define CHECK(c) do { if (!(c)) { std::printf("%s, line %d\n", #c, __LINE__); std::exit(1); } } while (0)

static void apply(const std::vector<CopyTask>& tasks, const Vec& src, Vec& dst) {
  for (const CopyTask& t : tasks)
    for (int64_t e = 0; e < t.numel(); ++e) {
      int64_t q = e, s = t.soff, d = t.doff;
      for (int i = 0; i < t.nd; ++i) {
        s += q % t.ext[i] * t.sstr[i];
        d += q % t.ext[i] * t.dstr[i];
        q /= t.ext[i];
      }
      dst[d] = src[s];
    }
}

static Vec fused(const Vec& a, const Vec& b, const ContractPlan& p) {
  Vec fa(p.fa.out.total), fb(p.fb.out.total), fc(p.mm.out.total, 0), c(p.split.out.total, -1);
  apply(p.fa.tasks, a, fa);
  apply(p.fb.tasks, b, fb);
  for (const GemmTask& g : p.mm.gemms)
    for (int64_t n = 0; n < g.N; ++n)
      for (int64_t m = 0; m < g.M; ++m) {
        int64_t s = 0;
        for (int64_t k = 0; k < g.K; ++k) s += fa[g.offA + m + k * g.lda] * fb[g.offB + k + n * g.ldb];
        fc[g.offC + m + n * g.ldc] = s;
      }
  apply(p.split.tasks, fc, c);
  return c;
}

// tensors of several parts, addressed as kernels do: part in the bits of the address
struct Parts {
  std::vector<Vec> v;
  int64_t& at(int64_t x) {
    return v.at((uint64_t)x >> kPartShift).at(x & (((int64_t)1 << kPartShift) - 1));
  }
};
static int64_t off(const int32_t* i, const int32_t* s) {
  int64_t o = 0;
  for (int d = 0; d < kMapLegs; ++d) o += (int64_t)i[d] * s[d];
  CHECK(o < ((int64_t)1 << 31));
  return o;
}
static int64_t at(const MapBlock& b, const AxisEntry& r, const AxisEntry& c) {
  return b.base + off(r.i, b.rs) + off(c.i, b.cs);
}
static int combo(const AxisEntry& e) { return e.combo_run & kComboMask; }

struct Sim {
  Parts A, B, C, written;
  void put(int64_t x, int64_t v) {
    C.at(x) = v;
    CHECK(++written.at(x) == 1);
  }
  void small(const DirectTables& t) {
    int64_t first = 0;
    for (const SmallProblem& s : t.small) {
      CHECK(s.first == first && s.mt == (s.M + 31) / 32);
      first += (int64_t)s.mt * ((s.N + 3) / 4);
      for (int i = 0; i < s.M; ++i)
        for (int j = 0; j < s.N; ++j) {
          const AxisEntry &x = t.axes.at(s.axM + i), &y = t.axes.at(s.axN + j);
          int64_t sum = 0;
          for (int k = 0; k < s.K; ++k) {
            const AxisEntry& z = t.axes.at(s.axK + k);
            sum += A.at(at(t.blocks.at(s.blkA + combo(x) * s.nkc + combo(z)), x, z)) *
                   B.at(at(t.blocks.at(s.blkB + combo(y) * s.nkc + combo(z)), y, z));
          }
          put(at(t.blocks.at(s.blkC + combo(x) * s.nnc + combo(y)), x, y), sum);
        }
    }
    CHECK(first == t.small_tiles);
  }
  void thin(const DirectTables& t) {
    int last = 1 << 30;
    for (const ThinUnit& u : t.units) {
      CHECK(u.count <= last && u.T <= kThinMax && u.K <= kThinMax);
      last = u.count;
      Parts &L = u.longB ? B : A, &S = u.longB ? A : B;
      for (int r = 0; r < u.count; ++r) {
        const uint32_t q = u.start + r, q0 = fdiv(q, u.m0, u.s0), q1 = fdiv(q0, u.m1, u.s1);
        const int32_t i[3] = {(int32_t)(q - q0 * u.d0), (int32_t)(q0 - q1 * u.d1), (int32_t)q1};
        auto where = [&](const ThinOffset& o) {
          const int32_t s[3] = {o.rs0, o.rs1, o.rs2};
          return o.off + off(i, s);
        };
        for (int y = 0; y < u.T; ++y) {
          int64_t sum = 0;
          for (int k = 0; k < u.K; ++k)
            sum += L.at(where(t.offs.at(u.offs + k))) * S.at(t.vals.at(u.vals + y * u.K + k));
          put(where(t.offs.at(u.offs + u.K + y)), sum);
        }
      }
    }
  }
  void tiled(const DirectTables& d, int sms, int* cut, int* swapped) {
    using namespace f64tc;
    if (d.tiled.empty()) return;
    Group G;
    GroupTables t;
    plan_group(d.tiled, sms, G, t);
    check_group(d.tiled, G, t, cut, swapped);
    for (const Problem& P : t.probs) {
      Parts &R = P.swap ? B : A, &S = P.swap ? A : B;
      for (int64_t m = 0; m < P.M; ++m)
        for (int64_t n = 0; n < P.N; ++n) {
          const AxisEntry &x = t.axes.at(P.axM + m), &y = t.axes.at(P.axN + n);
          int64_t sum = 0;
          for (int64_t k = 0; k < P.K; ++k) {
            const AxisEntry& z = t.axes.at(P.axK + k);
            sum += R.at(at(t.blocks.at(P.blkA + combo(x) * P.nkc + combo(z)), x, z)) *
                   S.at(at(t.blocks.at(P.blkB + combo(y) * P.nkc + combo(z)), y, z));
          }
          put(at(t.blocks.at(P.blkC + combo(x) * P.nnc + combo(y)), x, y), sum);
        }
    }
  }
  // every output tile once, its pieces covering the K steps once, in an order of decreasing steps
  static void check_group(const std::vector<f64tc::Task>& tasks, const f64tc::Group& G,
                          const f64tc::GroupTables& t, int* cut, int* swapped) {
    using namespace f64tc;
    CHECK(G.nprob == (int)tasks.size() && t.probs.size() == tasks.size());
    CHECK(G.ntiles == (int64_t)t.tiles.size() && G.nitems == (int)t.items.size());
    std::map<std::array<int, 3>, std::vector<Tile>> by;
    int64_t with_k = 0;
    for (size_t i = 0; i < t.tiles.size(); ++i) {
      const Tile& x = t.tiles[i];
      by[{x.prob, x.mi, x.ni}].push_back(x);
      with_k += x.ks1 > x.ks0;
      if (i) CHECK(t.tiles[i - 1].ks1 - t.tiles[i - 1].ks0 >= x.ks1 - x.ks0);
    }
    CHECK(with_k == G.ntiles_k);
    std::set<int> slots;
    size_t ntiles = 0;
    int64_t tA = 0, tB = 0, lA = 0, lB = 0, rA = 0, rB = 0;
    for (size_t p = 0; p < t.probs.size(); ++p) {
      const Problem& P = t.probs[p];
      const GemmTask& g = tasks[p].g;
      *swapped += P.swap != 0;
      CHECK(P.M == (P.swap ? g.N : g.M) && P.N == (P.swap ? g.M : g.N) && P.K == g.K);
      CHECK(P.mt == (P.M + BM - 1) / BM && P.nt == (P.N + BN - 1) / BN && P.nk == (P.K + BK - 1) / BK);
      CHECK(P.tA == tA && P.tB == tB && P.lA == lA && P.lB == lB && P.rA == rA && P.rB == rB);
      tA += (int64_t)P.mt * P.nk, tB += (int64_t)P.nt * P.nk;
      lA += (P.M + 31) / 32, lB += (P.N + 31) / 32, rA += P.M, rB += P.N;
      for (int mi = 0; mi < P.mt; ++mi)
        for (int ni = 0; ni < P.nt; ++ni) {
          auto v = by[{(int)p, mi, ni}];
          CHECK(!v.empty());
          std::sort(v.begin(), v.end(), [](const Tile& a, const Tile& b) { return a.ks0 < b.ks0; });
          int ks = 0;
          for (const Tile& x : v) {
            CHECK(x.ks0 == ks && (x.ks1 > x.ks0 || P.nk == 0) && x.parts == (int)v.size());
            ks = x.ks1;
            CHECK(P.K <= 8000 || (x.ks1 - x.ks0) * BK <= 8000);  // sums of a piece fit 64 bits
            CHECK(x.K == P.K && x.slot == v[0].slot);
            CHECK(x.rowA == (P.tA + (int64_t)mi * P.nk) * BM && x.rowB == (P.tB + (int64_t)ni * P.nk) * BN);
            CHECK(x.lA == P.lA + mi * (BM / 32) && x.lB == P.lB + ni * (BN / 32));
            CHECK(x.nA == std::min<int64_t>(BM / 32, (P.M + 31) / 32 - mi * (BM / 32)) && x.nA > 0);
            CHECK(x.nB == std::min<int64_t>(BN / 32, (P.N + 31) / 32 - ni * (BN / 32)) && x.nB > 0);
          }
          CHECK(ks == P.nk);
          if (v.size() > 1) {
            ++*cut;
            CHECK(v[0].slot >= 0 && v[0].slot < G.nslots && slots.insert(v[0].slot).second);
          }
          ++ntiles;
        }
    }
    CHECK(by.size() == ntiles && (int64_t)slots.size() == G.nslots);
    CHECK(G.lA == lA && G.lB == lB && G.rA == rA && G.rB == rB);
    CHECK(G.rowsA >= tA * BM && G.rowsB >= tB * BN);
    std::set<std::array<int, 3>> items;
    for (const int2& it : t.items) {
      const Problem& P = t.probs.at(it.x & 0x3fffffff);
      const int side = it.x >> 30 & 1;
      CHECK(it.y % 32 == 0 && it.y < (side ? P.N : P.M) && P.K > 0);
      CHECK(items.insert({it.x & 0x3fffffff, side, it.y}).second);
    }
    size_t want = 0;
    for (const Problem& P : t.probs)
      if (P.K) want += (P.M + 31) / 32 + (P.N + 31) / 32;
    CHECK(items.size() == want);
  }
};

// fused problems of given sizes, for the cuts alone
static void cuts(std::mt19937& rng, int* cut) {
  auto uni = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  for (int round = 0; round < 50; ++round) {
    std::vector<f64tc::Task> g;
    int64_t at[3] = {0, 0, 0};
    for (int n = uni(1, 9); n; --n) {
      f64tc::Task x;
      const int big = uni(0, 3);
      x.g.M = uni(1, big == 1 ? 3000 : 200);
      x.g.N = uni(1, big == 2 ? 3000 : 200);
      x.g.K = uni(0, 9) ? uni(1, big == 3 ? 65536 : 900) : 0;
      x.g.lda = x.g.M, x.g.ldb = x.g.K, x.g.ldc = x.g.M;
      x.g.offA = at[0], x.g.offB = at[1], x.g.offC = at[2];
      g.push_back(x);
    }
    f64tc::Group G;
    f64tc::GroupTables t;
    const int sms[4] = {1, 4, 152, 1000};
    f64tc::plan_group(g, sms[uni(0, 3)], G, t);
    int swapped = 0;
    Sim::check_group(g, G, t, cut, &swapped);
  }
}

int main(int argc, char** argv) {
  std::mt19937 rng(std::atoi(argv[1]));
  auto uni = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  int nsmall = 0, nthin = 0, ntiled = 0, cut = 0, swapped = 0;
  for (int round = 0; round < 40; ++round) {
    const int kind = round % 4;  // small; one long axis; a long K; both axes wide
    const int ra = uni(1, 3), rb = uni(1, 3), nc = kind == 2 ? 1 : uni(1, 2);
    auto space = [&](int longest) {
      std::vector<std::pair<int, int64_t>> s;
      const int first = uni(-1, 1), n = uni(1, 3);
      for (int i = 0; i < n; ++i) s.push_back({first + i, uni(1, 4)});
      if (longest) s[uni(0, n - 1)].second = uni(longest / 2, longest);
      return Space::make(s, uni(0, 1));
    };
    std::vector<Space> con, sa, sb;
    std::vector<int> ia, ib, label;
    for (int i = 0; i < ra + rb; ++i) label.push_back(i + 1);
    std::shuffle(label.begin(), label.end(), rng);
    for (int i = 0; i < nc; ++i) con.push_back(space(i == 0 && kind >= 2 ? 540 : i == 0 && kind == 1 ? 12 : 0));
    const int la_long = kind == 3 || (kind == 1 && uni(0, 1)) ? uni(0, ra - 1) : -1;
    const int lb_long = kind == 3 || (kind == 1 && la_long < 0) ? uni(0, rb - 1) : -1;
    struct Leg { Space s; int idx; };
    std::vector<Leg> la, lb;
    for (int i = 0; i < nc; ++i) { la.push_back({con[i], -1 - i}); lb.push_back({dual_space(con[i]), -1 - i}); }
    for (int i = 0; i < ra; ++i) la.push_back({space(i == la_long ? (kind == 3 ? 90 : 60000) : 0), label[i]});
    for (int i = 0; i < rb; ++i) lb.push_back({space(i == lb_long ? (kind == 3 ? 90 : 60000) : 0), label[ra + i]});
    std::shuffle(la.begin(), la.end(), rng);
    std::shuffle(lb.begin(), lb.end(), rng);
    for (auto& l : la) { sa.push_back(l.s); ia.push_back(l.idx); }
    for (auto& l : lb) { sb.push_back(l.s); ib.push_back(l.idx); }
    const TensorMeta A = TensorMeta::build(uni(-1, 1), sa), B = TensorMeta::build(uni(-1, 1), sb);
    auto p = plan_contract(A, ia, B, ib);
    if (p->mm.flops > 1.6e7) continue;
    const bool ca = uni(0, 1), cb = uni(0, 1);
    auto map = build_contract_map(*p, A, B);
    CHECK(map.size() == p->mm.gemms.size());
    if (ca || cb) map = complex_map(map, ca, cb);
    std::vector<GemmTask> gemms = p->mm.gemms;
    for (GemmTask& g : gemms) { if (ca) g.M *= 2; if (cb) g.N *= 2; }
    Sim s;
    for (Parts* x : {&s.A, &s.B})
      for (int i = 0; i < ((x == &s.A ? ca : cb) ? 2 : 1); ++i) {
        Vec v((x == &s.A ? A : B).total);
        for (auto& e : v) e = uni(-9, 9);
        x->v.push_back(v);
      }
    const int np = (ca ? 2 : 1) * (cb ? 2 : 1);
    s.C.v.assign(np, Vec(p->split.out.total, -1));
    s.written.v.assign(np, Vec(p->split.out.total, 0));
    DirectTables t;
    const int sms = uni(0, 1) ? 152 : 3;
    plan_direct(map, gemms, sms, t);
    s.small(t);
    s.thin(t);
    s.tiled(t, sms, &cut, &swapped);
    nsmall += !t.small.empty(), nthin += !t.units.empty(), ntiled += !t.tiled.empty();
    for (int i = 0; i < np; ++i)  // part of the result: 2 [part of A] + [part of B], or the complex one's
      CHECK(s.C.v[i] == fused(s.A.v[cb ? i / 2 * ca : i], s.B.v[cb ? i % 2 : 0], *p));
  }
  cuts(rng, &cut);
  std::printf("ok %d %d %d %d %d\n", nsmall, nthin, ntiled, cut, swapped);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed")
def test_tables_cover_and_compute_every_contraction(tmp_path):
    import mps_gb300  # noqa: F401  (builds the library that the harness links)
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    lib = os.path.dirname(build.LIB)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-I", os.path.join(CUDA, "include"), str(src),
                    build.LIB, f"-Wl,-rpath,{lib}", "-L", os.path.join(CUDA, "lib64"), "-lcudart",
                    f"-Wl,-rpath,{os.path.join(CUDA, 'lib64')}", "-o", str(exe)], check=True)
    met = [0] * 5  # small, thin, tiled contractions; cut tiles; problems taken the other way round
    for seed in range(4):
        r = subprocess.run([str(exe), str(seed)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
        met = [a + int(b) for a, b in zip(met, r.stdout.split()[1:])]
    assert min(met) >= 2, met
