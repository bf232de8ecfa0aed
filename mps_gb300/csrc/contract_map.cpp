// Index maps of a contraction (see contract_map.hpp).
#include "contract_map.hpp"

#include <algorithm>
#include <map>
#include <unordered_map>

namespace mpsg {

namespace {

constexpr int64_t kMaxStride = (int64_t)1 << 31;

// A source block as a rectangle of a fused block.
struct Rect {
  int64_t r0, c0;  // first row and column in the fused block
  size_t block;    // block of the tensor
};

// Groups the blocks of a tensor by the fused block they belong to; map[b].off is the position of
// block b's first element in the fused buffer.
std::vector<std::vector<Rect>> rects_of(const TensorMeta& fused, const std::vector<BlockMap>& map) {
  std::vector<std::vector<Rect>> out(fused.nblocks());
  for (size_t b = 0; b < map.size(); ++b) {
    const auto it = std::upper_bound(fused.off.begin(), fused.off.end(), map[b].off);
    const size_t f = (size_t)(it - fused.off.begin()) - 1;
    const int64_t rel = map[b].off - fused.off[f], rows = fused.sec.sizes(f)[0];
    out[f].push_back(Rect{rel % rows, rel / rows, b});
  }
  return out;
}

// The combos of one side of a fused block from its rectangles: starts, and leg sizes `legs` of
// the block that has each start. False when two blocks disagree.
bool combos_of(const std::vector<Rect>& rects, bool rows, const TensorMeta& T,
               const std::vector<int>& legs, std::vector<AxisCombo>& out) {
  std::map<int64_t, AxisCombo> at;
  for (const Rect& r : rects) {
    AxisCombo c;
    c.start = (int32_t)(rows ? r.r0 : r.c0);
    int64_t n = 1;
    for (int d = 0; d < kMapLegs; ++d) {
      const int64_t z = d < (int)legs.size() ? T.sec.sizes(r.block)[legs[d]] : 1;
      c.d[d] = (int32_t)z;
      n *= z;
    }
    c.count = (int32_t)n;
    auto ins = at.emplace(c.start, c);
    const AxisCombo& o = ins.first->second;
    if (o.count != c.count || !std::equal(o.d, o.d + kMapLegs, c.d)) return false;
  }
  int64_t next = 0;
  out.clear();
  for (auto& kv : at) {
    if (kv.first != next) return false;
    next += kv.second.count;
    out.push_back(kv.second);
  }
  return true;
}

bool same_combos(const std::vector<AxisCombo>& a, const std::vector<AxisCombo>& b) {
  if (a.size() != b.size()) return false;
  for (size_t i = 0; i < a.size(); ++i)
    if (a[i].start != b[i].start || a[i].count != b[i].count ||
        !std::equal(a[i].d, a[i].d + kMapLegs, b[i].d))
      return false;
  return true;
}

size_t combo_at(const std::vector<AxisCombo>& c, int64_t start) {
  size_t lo = 0, hi = c.size();
  while (hi - lo > 1) {
    const size_t mid = (lo + hi) / 2;
    (c[mid].start <= start ? lo : hi) = mid;
  }
  return lo;
}

// Block table [major combo][minor combo]; the major axis is the rectangles' rows unless
// `transposed`. False when a combination is missing or twice there, or a stride is too long.
bool table_of(const std::vector<Rect>& rects, const TensorMeta& T, const std::vector<int>& row_legs,
              const std::vector<int>& col_legs, const std::vector<AxisCombo>& rows,
              const std::vector<AxisCombo>& cols, bool transposed, std::vector<MapBlock>& out) {
  const size_t nr = rows.size(), nc = cols.size();
  if (rects.size() != nr * nc) return false;
  std::vector<char> seen(nr * nc, 0);
  out.assign(nr * nc, MapBlock());
  for (const Rect& r : rects) {
    const size_t i = combo_at(rows, r.r0), j = combo_at(cols, r.c0);
    const size_t at = transposed ? j * nr + i : i * nc + j;
    if (seen[at]) return false;
    seen[at] = 1;
    int64_t str[kMaxLegs], s = 1;
    for (int k = 0; k < T.N(); ++k) {
      str[k] = s;
      s *= T.sec.sizes(r.block)[k];
    }
    if (s >= kMaxStride) return false;  // offsets within a block are 32-bit
    MapBlock& b = out[at];
    b.base = T.off[r.block];
    for (int d = 0; d < kMapLegs; ++d) {
      const int64_t x = d < (int)row_legs.size() ? str[row_legs[d]] : 0;
      const int64_t y = d < (int)col_legs.size() ? str[col_legs[d]] : 0;
      if (x >= kMaxStride || y >= kMaxStride) return false;
      b.rs[d] = (int32_t)(transposed ? y : x);
      b.cs[d] = (int32_t)(transposed ? x : y);
    }
  }
  return true;
}

// Makes the longest leg of an axis its leg 0, in the combos and in the tables that use the axis.
void longest_first(std::vector<AxisCombo>& axis, std::vector<MapBlock>* t1, bool rows1,
                   std::vector<MapBlock>* t2, bool rows2) {
  int32_t len[kMapLegs] = {0, 0, 0};
  for (const AxisCombo& c : axis)
    for (int d = 0; d < kMapLegs; ++d) len[d] = std::max(len[d], c.d[d]);
  const int best = (int)(std::max_element(len, len + kMapLegs) - len);
  if (best == 0) return;
  for (AxisCombo& c : axis) std::swap(c.d[0], c.d[best]);
  for (MapBlock& b : *t1) std::swap((rows1 ? b.rs : b.cs)[0], (rows1 ? b.rs : b.cs)[best]);
  for (MapBlock& b : *t2) std::swap((rows2 ? b.rs : b.cs)[0], (rows2 ? b.rs : b.cs)[best]);
}

std::vector<int> zero_based(const std::vector<int>& v) {
  std::vector<int> o;
  for (int x : v) o.push_back(x - 1);
  return o;
}

}  // namespace

void append_axis(const std::vector<AxisCombo>& combos, std::vector<AxisEntry>& out) {
  for (size_t c = 0; c < combos.size(); ++c) {
    const int32_t* d = combos[c].d;
    for (int32_t z = 0; z < d[2]; ++z)
      for (int32_t y = 0; y < d[1]; ++y)
        for (int32_t x = 0; x < d[0]; ++x)
          out.push_back(AxisEntry{(int32_t)c | std::min(d[0] - x, 255) << 24, {x, y, z}});
  }
}

std::vector<MapProblem> complex_map(const std::vector<MapProblem>& map, bool ca, bool cb) {
  std::vector<MapProblem> out;
  auto twice = [](std::vector<AxisCombo>& axis, int64_t n) {
    const size_t k = axis.size();
    for (size_t i = 0; i < k; ++i) {
      axis.push_back(axis[i]);
      axis.back().start += (int32_t)n;
    }
  };
  auto with_part = [](std::vector<MapBlock>& t) {
    const size_t k = t.size();
    for (size_t i = 0; i < k; ++i) {
      t.push_back(t[i]);
      t.back().base |= (int64_t)1 << kPartShift;
    }
  };
  for (MapProblem q : map) {
    const size_t nm = q.m.size(), nn = q.n.size();
    const std::vector<MapBlock> c = q.C;
    const int pa = ca ? 2 : 1, pb = cb ? 2 : 1;
    if (q.M * pa > INT32_MAX || q.N * pb > INT32_MAX ||
        std::max(nm * pa, nn * pb) > (size_t)kComboMask)
      return {};
    q.C.clear();
    for (int x = 0; x < pa; ++x)
      for (size_t i = 0; i < nm; ++i)
        for (int y = 0; y < pb; ++y)
          for (size_t j = 0; j < nn; ++j) {
            q.C.push_back(c[i * nn + j]);
            q.C.back().base |= (int64_t)(x * pb + y) << kPartShift;
          }
    if (ca) {
      twice(q.m, q.M);
      with_part(q.A);
      q.M *= 2;
    }
    if (cb) {
      twice(q.n, q.N);
      with_part(q.B);
      q.N *= 2;
    }
    out.push_back(std::move(q));
  }
  return out;
}

std::vector<MapProblem> build_contract_map(const ContractPlan& p, const TensorMeta& A,
                                           const TensorMeta& B) {
  std::vector<MapProblem> none;
  if (p.scalar) return none;
  const std::vector<int> ra = zero_based(p.rowsA), ka = zero_based(p.colsA),
                         kb = zero_based(p.rowsB), cb = zero_based(p.colsB);
  if ((int)std::max(std::max(ra.size(), ka.size()), cb.size()) > kMapLegs) return none;
  // axes of the result that hold A's and B's open legs, in fused order
  std::vector<int> rc(ra.size()), cc(cb.size());
  for (size_t j = 0; j < p.perm.size(); ++j) {
    const size_t leg = (size_t)p.perm[j] - 1;
    (leg < ra.size() ? rc[leg] : cc[leg - ra.size()]) = (int)j;
  }
  std::vector<BlockMap> ma, mb, mc;
  plan_symmatrix_rec(A, p.rowsA, p.colsA, &ma);
  plan_symmatrix_rec(B, p.rowsB, p.colsB, &mb);
  plan_split_permute_rec(p.mm.out, p.rlegs, p.clegs, p.perm, &mc);
  const auto fa = rects_of(p.fa.out, ma), fb = rects_of(p.fb.out, mb),
             fc = rects_of(p.mm.out, mc);
  std::unordered_map<int64_t, size_t> ata, atb, atc;
  for (size_t f = 0; f < p.fa.out.nblocks(); ++f) ata[p.fa.out.off[f]] = f;
  for (size_t f = 0; f < p.fb.out.nblocks(); ++f) atb[p.fb.out.off[f]] = f;
  for (size_t f = 0; f < p.mm.out.nblocks(); ++f) atc[p.mm.out.off[f]] = f;
  std::vector<MapProblem> out;
  const TensorMeta& C = p.split.out;
  for (const GemmTask& g : p.mm.gemms) {
    MapProblem q;
    q.M = g.M;
    q.N = g.N;
    q.K = g.K;
    if (g.M > INT32_MAX || g.N > INT32_MAX || g.K > INT32_MAX) return none;
    const auto ic = atc.find(g.offC);
    if (ic == atc.end()) return none;
    const auto& rects_c = fc[ic->second];
    if (!combos_of(rects_c, true, C, rc, q.m) || !combos_of(rects_c, false, C, cc, q.n) ||
        !table_of(rects_c, C, rc, cc, q.m, q.n, false, q.C))
      return none;
    if (g.K > 0) {
      const auto ia = ata.find(g.offA), ib = atb.find(g.offB);
      if (ia == ata.end() || ib == atb.end()) return none;
      const auto &rects_a = fa[ia->second], &rects_b = fb[ib->second];
      std::vector<AxisCombo> m, k, n;
      if (!combos_of(rects_a, true, A, ra, m) || !combos_of(rects_a, false, A, ka, q.k) ||
          !combos_of(rects_b, true, B, kb, k) || !combos_of(rects_b, false, B, cb, n) ||
          !same_combos(m, q.m) || !same_combos(n, q.n) || !same_combos(k, q.k) ||
          !table_of(rects_a, A, ra, ka, q.m, q.k, false, q.A) ||
          !table_of(rects_b, B, kb, cb, q.k, q.n, true, q.B))
        return none;
    }
    if (std::max(std::max(q.m.size(), q.n.size()), q.k.size()) > (size_t)kComboMask) return none;
    longest_first(q.m, &q.A, true, &q.C, true);
    longest_first(q.n, &q.B, true, &q.C, false);
    longest_first(q.k, &q.A, false, &q.B, false);
    out.push_back(std::move(q));
  }
  return out;
}

}  // namespace mpsg
