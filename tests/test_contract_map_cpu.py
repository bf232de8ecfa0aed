"""Index maps of a contraction (mps_gb300/csrc/contract_map.cpp) on the CPU, compiled with g++: for
random structures, the sector GEMMs taken through the maps give, in integers, what fusing the
operands, multiplying and splitting the result give through the planner's copy tasks."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mps_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include "contract_map.hpp"
using namespace mpsg;
typedef std::vector<int64_t> Vec;

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

static int64_t at(const MapBlock& b, const AxisEntry& r, const AxisEntry& c) {
  int64_t o = b.base;
  for (int d = 0; d < kMapLegs; ++d) o += (int64_t)r.i[d] * b.rs[d] + (int64_t)c.i[d] * b.cs[d];
  return o;
}

static std::vector<AxisEntry> axis(const std::vector<AxisCombo>& c, int64_t n) {
  std::vector<AxisEntry> e;
  append_axis(c, e);
  if ((int64_t)e.size() != n) { std::printf("axis length\n"); std::exit(1); }
  for (size_t i = 0; i < e.size(); ++i) {
    const int run = (int)((uint32_t)e[i].combo_run >> 24);
    if (run < 1 || i + run > e.size()) { std::printf("run\n"); std::exit(1); }
    for (int r = 1; r < run; ++r) {
      const AxisEntry &x = e[i], &y = e[i + r];
      if ((x.combo_run & kComboMask) != (y.combo_run & kComboMask) || y.i[0] != x.i[0] + r ||
          y.i[1] != x.i[1] || y.i[2] != x.i[2]) { std::printf("run entries\n"); std::exit(1); }
    }
  }
  return e;
}

static Vec mapped(const Vec& a, const Vec& b, const ContractPlan& p, const std::vector<MapProblem>& map) {
  Vec c(p.split.out.total, -1);
  for (const MapProblem& q : map) {
    const auto m = axis(q.m, q.M), n = axis(q.n, q.N), k = axis(q.k, q.K);
    const size_t nk = q.k.size(), nn = q.n.size();
    for (const AxisEntry& x : m)
      for (const AxisEntry& y : n) {
        const int xc = x.combo_run & kComboMask, yc = y.combo_run & kComboMask;
        int64_t s = 0;
        for (const AxisEntry& z : k) {
          const int zc = z.combo_run & kComboMask;
          s += a.at(at(q.A[xc * nk + zc], x, z)) * b.at(at(q.B[yc * nk + zc], y, z));
        }
        c.at(at(q.C[xc * nn + yc], x, y)) = s;
      }
  }
  return c;
}

int main(int argc, char** argv) {
  std::mt19937 rng(std::atoi(argv[1]));
  auto uni = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
  int mapped_count = 0, wide = 0;
  for (int round = 0; round < 60; ++round) {
    const int ra = uni(1, 4), rb = uni(1, 3), nc = uni(1, 3);
    auto space = [&] {
      std::vector<std::pair<int, int64_t>> s;
      const int first = uni(-1, 1), n = uni(1, 3);
      for (int i = 0; i < n; ++i) s.push_back({first + i, uni(1, 4)});
      return Space::make(s, uni(0, 1));
    };
    std::vector<Space> con, sa, sb;
    std::vector<int> ia, ib, label;
    for (int i = 0; i < ra + rb; ++i) label.push_back(i + 1);
    std::shuffle(label.begin(), label.end(), rng);
    for (int i = 0; i < nc; ++i) con.push_back(space());
    struct Leg { Space s; int idx; };
    std::vector<Leg> la, lb;
    for (int i = 0; i < nc; ++i) { la.push_back({con[i], -1 - i}); lb.push_back({dual_space(con[i]), -1 - i}); }
    for (int i = 0; i < ra; ++i) la.push_back({space(), label[i]});
    for (int i = 0; i < rb; ++i) lb.push_back({space(), label[ra + i]});
    std::shuffle(la.begin(), la.end(), rng);
    std::shuffle(lb.begin(), lb.end(), rng);
    for (auto& l : la) { sa.push_back(l.s); ia.push_back(l.idx); }
    for (auto& l : lb) { sb.push_back(l.s); ib.push_back(l.idx); }
    const TensorMeta A = TensorMeta::build(uni(-1, 1), sa), B = TensorMeta::build(uni(-1, 1), sb);
    auto p = plan_contract(A, ia, B, ib);
    const auto map = build_contract_map(*p, A, B);
    if (ra > kMapLegs) { if (!map.empty()) { std::printf("too many legs mapped\n"); return 1; } ++wide; continue; }
    if (map.size() != p->mm.gemms.size()) { std::printf("not mapped\n"); return 1; }
    Vec a(A.total), b(B.total);
    for (auto& x : a) x = uni(-9, 9);
    for (auto& x : b) x = uni(-9, 9);
    if (fused(a, b, *p) != mapped(a, b, *p, map)) { std::printf("round %d differs\n", round); return 1; }
    mapped_count += p->split.out.total > 0;
  }
  std::printf("ok %d mapped, %d with too many legs\n", mapped_count, wide);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed")
def test_maps_equal_the_copy_tasks(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text("#include <algorithm>\n" + HARNESS)
    exe = tmp_path / "harness"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src),
                    os.path.join(CSRC, "planner.cpp"), os.path.join(CSRC, "contract_map.cpp"), "-o",
                    str(exe)], check=True)
    for seed in range(4):
        r = subprocess.run([str(exe), str(seed)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        assert r.stdout.startswith("ok"), r.stdout
