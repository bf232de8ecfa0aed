// Sector GEMMs of a contraction on the FP64 pipe, reading the operand tensors and writing the result
// tensor in place through index maps (contract_map.hpp): the element-per-thread kernel for small
// contractions and the thin kernel for MPO-sized ones. The large sector GEMMs take the same maps
// into the tensor-core kernels (kernels_f64tc.cu).
#include <algorithm>

#include "copy_decode.hpp"
#include "dep_load.cuh"
#include "direct.hpp"

namespace mpsg {

namespace {

struct BlockRegs {
  int64_t base;
  int rs0, rs1, rs2, cs0, cs1, cs2;
};

__device__ __forceinline__ BlockRegs load_block(const MapBlock* b, int64_t d1, int64_t d2 = 0,
                                                int64_t d3 = 0) {
  const int4* p = reinterpret_cast<const int4*>(b);
  const int4 x = __ldg(p), y = __ldg(p + 1);
  const int64_t base = (int64_t)(((unsigned long long)(unsigned)x.y << 32) | (unsigned)x.x);
  return BlockRegs{part_base(base, d1, d2, d3), x.z, x.w, y.x, y.y, y.z, y.w};
}

__device__ __forceinline__ int64_t row_part(const BlockRegs& b, const int4& e) {
  return b.base + (e.y * b.rs0 + e.z * b.rs1 + e.w * b.rs2);
}

__device__ __forceinline__ int col_part(const BlockRegs& b, const int4& e) {
  return e.y * b.cs0 + e.z * b.cs1 + e.w * b.cs2;
}

// Every sector GEMM of a small contraction in one launch: a CTA takes 32 rows and 4 columns of a result,
// one element per thread, its operands staged in shared memory kChunk contracted indices at a
// time. Bound by latency: what counts is that the elements spread over the whole chip (a 64 x 64 tile
// kernel keeps them on a few SMs, each at 2 FMAs per cycle), that the loads of an element's sum do
// not wait for one another (all of a CTA's are issued at once, index tables first; as a loop of
// each thread they took 15 of the last contraction's 17 us) and that nothing runs before or after it.
// Measured, the four contractions of a chi = 48 two-site H_eff: 26.6 us with the gaps between them (29.7 us as thread loops) against
// 19 launches of 205 us in all.
constexpr int kChunk = 128, kSmallRows = 32, kSmallCols = 4;

// Offset of a row's (or column's) element at contracted index x, through its block table.
__device__ __forceinline__ int64_t mapped_at(const MapBlock* __restrict__ tab, const int4& row,
                                             const int4& x, int64_t d1) {
  const BlockRegs b = load_block(tab + (x.x & kComboMask), d1);
  return row_part(b, row) + col_part(b, x);
}

__global__ void __launch_bounds__(kSmallRows * kSmallCols) contract_small_kernel(
    const SmallProblem* __restrict__ probs, int nprob, int ntiles,
    const AxisEntry* __restrict__ axes, const MapBlock* __restrict__ blocks,
    const double* A, const double* B, double* __restrict__ C,
    const PartOffsets parts) {
  __shared__ double as[kChunk * kSmallRows], bs[kChunk * kSmallCols];
  const int4* ax = reinterpret_cast<const int4*>(axes);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  cudaTriggerProgrammaticLaunchCompletion();
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(&probs[mid].first) <= tile) lo = mid;
      else hi = mid - 1;
    }
    const SmallProblem P = probs[lo];
    const int ni = (tile - P.first) / P.mt, mi = tile - P.first - ni * P.mt;
    const int i = mi * kSmallRows + lane, j = ni * kSmallCols + w;
    const int4 me = __ldg(ax + P.axM + min(i, P.M - 1)), ne = __ldg(ax + P.axN + min(j, P.N - 1));
    const int4 nl = __ldg(ax + P.axN + min(ni * kSmallCols + (t & 3), P.N - 1));  // column it stages
    const MapBlock* ta = blocks + P.blkA + (me.x & kComboMask) * P.nkc;
    const MapBlock* tb = blocks + P.blkB + (nl.x & kComboMask) * P.nkc;
    const BlockRegs bc =
        load_block(blocks + P.blkC + (me.x & kComboMask) * P.nnc + (ne.x & kComboMask), parts.c1,
                   parts.c2, parts.c3);
    double acc = 0.0;
    for (int c0 = 0; c0 == 0 || c0 < P.K; c0 += kChunk) {
      const int4* ke = ax + P.axK + c0;
      const int kn = min(kChunk, P.K - c0);
      constexpr int kPart = kChunk / 2, kA = kPart / kSmallCols, kB = kChunk / kSmallRows;
      int64_t oa[kA], ob[kB];  // all addresses, then all loads
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int k = (t >> 2) + kSmallRows * u;
        if (k < kn) ob[u] = mapped_at(tb, nl, __ldg(ke + k), parts.b);
      }
#pragma unroll
      for (int u = 0; u < kA; ++u) {
        const int k = w + kSmallCols * u;
        if (k < kn) oa[u] = mapped_at(ta, me, __ldg(ke + k), parts.a);
      }
      if (tile == blockIdx.x && c0 == 0) cudaGridDependencySynchronize();
      double va[kA], vb[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u)
        if ((t >> 2) + kSmallRows * u < kn) vb[u] = load_dep(B + ob[u]);
#pragma unroll
      for (int u = 0; u < kA; ++u)
        if (w + kSmallCols * u < kn) va[u] = load_dep(A + oa[u]);
      if (c0 > 0 || tile != blockIdx.x) __syncthreads();  // the last chunk has been read
#pragma unroll
      for (int u = 0; u < kA; ++u)
        if (w + kSmallCols * u < kn) as[(w + kSmallCols * u) * kSmallRows + lane] = va[u];
      if (kn > kPart) {
#pragma unroll
        for (int u = 0; u < kA; ++u) {
          const int k = kPart + w + kSmallCols * u;
          if (k < kn) va[u] = load_dep(A + mapped_at(ta, me, __ldg(ke + k), parts.a));
        }
#pragma unroll
        for (int u = 0; u < kA; ++u) {
          const int k = kPart + w + kSmallCols * u;
          if (k < kn) as[k * kSmallRows + lane] = va[u];
        }
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int k = (t >> 2) + kSmallRows * u;
        if (k < kn) bs[k * kSmallCols + (t & 3)] = vb[u];
      }
      __syncthreads();
#pragma unroll 8
      for (int k = 0; k < kn; ++k)
        acc = fma(as[k * kSmallRows + lane], bs[k * kSmallCols + w], acc);
    }
    if (i < P.M && j < P.N) C[row_part(bc, me) + col_part(bc, ne)] = acc;
  }
}

// Thin sector GEMMs (the MPO steps: T and K at most 32): a thread owns indices of the long axis,
// reads the K elements of each and writes T results, coalesced along the long axis; the thin
// operand sits in shared memory. Bound by the FP64 pipe (2 FMAs per SM and cycle) and HBM about
// equally for the XXZ MPO (K = T = 4), so FMAs with an exact zero of the thin operand are skipped
// (12 of its 34 allowed entries are not zero), a first term of 1.0 x is taken as x, and
// several rows are in flight per thread. A row with a non-finite element does every FMA, as 0 x Inf
// must give NaN. Measured, the MPO steps of a two-site H_eff with the copies that they replace:
// chi = 2048 2 x 41 us (before 434), chi = 517 2 x 11 us (93), each with four rows in flight per thread
// (launch_direct has the whole application with two, the faster choice).
struct ThinShared {
  ThinOffset o[2 * kThinMax];    // K of the long operand, T of the output
  uint32_t mask[kThinMax];       // nonzero entries of a thin index
  uint32_t one[kThinMax];        // its lowest nonzero entry if that is exactly 1.0
  double b[kThinMax * kThinMax];  // [thin][k]
};

// x as fma(x, 1.0, 0.0) gives it: -0.0 becomes 0.0
__device__ __forceinline__ double times_one(double x) {
  const long long b = __double_as_longlong(x);
  return __longlong_as_double(b == (long long)(1ull << 63) ? 0 : b);
}

// acc += the terms of entries k0 .. k0 + 3 in the low four bits of PAT; bit 4: the first of them starts
// the sum and its factor is 1.0.
template <int PAT, int KMAX, int ROWS>
__device__ __forceinline__ void thin_terms(double (&acc)[ROWS], const double (&a)[ROWS][KMAX],
                                           int k0, const double* b) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!(PAT >> k & 1)) continue;
    if (PAT >> 4 && (PAT & ((1 << k) - 1)) == 0) {
#pragma unroll
      for (int y = 0; y < ROWS; ++y) acc[y] = times_one(a[y][k0 + k]);
    } else {
      const double f = b[k0 + k];
#pragma unroll
      for (int y = 0; y < ROWS; ++y) acc[y] = fma(a[y][k0 + k], f, acc[y]);
    }
  }
}

// ROWS groups of 32 rows, one row of each per lane, from `row` on (all groups below u.count begin
// inside the unit).
template <int KMAX, int ROWS>
__device__ __forceinline__ void thin_rows(const ThinShared& s, const ThinUnit& u, int row,
                                          const double* X, double* __restrict__ C) {
  const int K = u.K;
  int i0[ROWS], i1[ROWS], i2[ROWS];
  bool in[ROWS];
  double a[ROWS][KMAX];
#pragma unroll
  for (int y = 0; y < ROWS; ++y) {
    in[y] = row + 32 * y < u.count;
    const uint32_t q = (uint32_t)(u.start + (in[y] ? row + 32 * y : 0));
    const uint32_t q0 = fdiv(q, u.m0, u.s0);
    i0[y] = (int)(q - q0 * u.d0);
    i2[y] = (int)fdiv(q0, u.m1, u.s1);
    i1[y] = (int)(q0 - (uint32_t)i2[y] * u.d1);
  }
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k < K) {
      const ThinOffset o = s.o[k];
#pragma unroll
      for (int y = 0; y < ROWS; ++y)
        a[y][k] = load_dep(X + o.off + (i0[y] * o.rs0 + i1[y] * o.rs1 + i2[y] * o.rs2));
    } else {
#pragma unroll
      for (int y = 0; y < ROWS; ++y) a[y][k] = 0.0;
    }
  }
  int bad = 0;
#pragma unroll
  for (int y = 0; y < ROWS; ++y)
#pragma unroll
    for (int k = 0; k < KMAX; ++k) bad |= (__double2hiint(a[y][k]) & 0x7ff00000) == 0x7ff00000;
  for (int t = 0; t < u.T; ++t) {
    const uint32_t mask = bad ? (K == 32 ? 0xffffffffu : (1u << K) - 1u) : s.mask[t];
    const uint32_t one = bad ? 0u : s.one[t];
    double acc[ROWS];
#pragma unroll
    for (int y = 0; y < ROWS; ++y) acc[y] = 0.0;
    // A jump per four entries: an FP64 instruction whose predicate is off still takes its slot of
    // the pipe; with conditional FMAs a step of the chi = 2048 H_eff took 72 us, with jumps 41.
#pragma unroll
    for (int k0 = 0; k0 < KMAX; k0 += 4) {
#define MPSG_THIN(P)                                          \
  case P:                                                     \
    thin_terms<P, KMAX, ROWS>(acc, a, k0, s.b + t * K);       \
    break;
      switch ((mask >> k0 & 15u) | ((one >> k0 & 15u) ? 16u : 0u)) {
        MPSG_THIN(1) MPSG_THIN(2) MPSG_THIN(3) MPSG_THIN(4) MPSG_THIN(5) MPSG_THIN(6) MPSG_THIN(7)
        MPSG_THIN(8) MPSG_THIN(9) MPSG_THIN(10) MPSG_THIN(11) MPSG_THIN(12) MPSG_THIN(13)
        MPSG_THIN(14) MPSG_THIN(15) MPSG_THIN(17) MPSG_THIN(18) MPSG_THIN(19) MPSG_THIN(20)
        MPSG_THIN(21) MPSG_THIN(22) MPSG_THIN(23) MPSG_THIN(24) MPSG_THIN(25) MPSG_THIN(26)
        MPSG_THIN(27) MPSG_THIN(28) MPSG_THIN(29) MPSG_THIN(30) MPSG_THIN(31)
        default:
          break;
      }
#undef MPSG_THIN
    }
    const ThinOffset o = s.o[K + t];
#pragma unroll
    for (int y = 0; y < ROWS; ++y)
      if (in[y]) C[o.off + (i0[y] * o.rs0 + i1[y] * o.rs1 + i2[y] * o.rs2)] = acc[y];
  }
}

template <int KMAX, int ROWS>
__global__ void __launch_bounds__(256) contract_thin_kernel(
    const ThinUnit* __restrict__ units, int nunits, const ThinOffset* __restrict__ offs,
    const int64_t* __restrict__ vals, const double* A, const double* B,
    double* __restrict__ C, const PartOffsets parts) {
  __shared__ ThinShared s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  cudaTriggerProgrammaticLaunchCompletion();
  for (int it = blockIdx.x; it < nunits; it += gridDim.x) {
    const ThinUnit u = units[it];
    const double* L = u.longB ? B : A;
    const double* S = u.longB ? A : B;
    __syncthreads();  // the previous unit has been read
    if (threadIdx.x < u.K + u.T) {
      ThinOffset o = offs[u.offs + threadIdx.x];
      o.off = threadIdx.x < u.K ? part_base(o.off, u.longB ? parts.b : parts.a, 0, 0)
                                : part_base(o.off, parts.c1, parts.c2, parts.c3);
      s.o[threadIdx.x] = o;
    }
    if (it == blockIdx.x) cudaGridDependencySynchronize();
    for (int x = threadIdx.x; x < u.T * u.K; x += blockDim.x)
      s.b[x] =
          load_dep(S + part_base(__ldg(vals + u.vals + x), u.longB ? parts.a : parts.b, 0, 0));
    __syncthreads();
    if (threadIdx.x < u.T) {
      const double* b = s.b + threadIdx.x * u.K;
      uint32_t m = 0;
      for (int k = 0; k < u.K; ++k) m |= (uint32_t)(__double_as_longlong(b[k]) << 1 != 0) << k;
      s.mask[threadIdx.x] = m;
      s.one[threadIdx.x] =
          m && __double_as_longlong(b[__ffs(m) - 1]) == 0x3ff0000000000000ll ? m & (0u - m) : 0u;
    }
    __syncthreads();
    // rows of a warp are 32 ROWS in a row; at the end of the unit the warps take 32 each
    const int full = u.count / (256 * ROWS) * (256 * ROWS);
    for (int r = 32 * ROWS * warp; r < full; r += 256 * ROWS)
      thin_rows<KMAX, ROWS>(s, u, r + lane, L, C);
    if (ROWS > 1)
      for (int r = full + 32 * warp; r < u.count; r += 256) thin_rows<KMAX, 1>(s, u, r + lane, L, C);
    else if (full + 32 * warp < u.count)
      thin_rows<KMAX, ROWS>(s, u, full + 32 * warp + lane, L, C);
  }
}

// FMAs of a contraction that stays element-per-thread: 2^21 take the FP64 pipes of 152 SMs 3.5 us when
// spread evenly, the tensor-core pair of launches about 20 us for anything.
constexpr int64_t kSmallFma = 1 << 21;
constexpr int64_t kSmallAxes = 1 << 16;  // ... and its axis entries (16 bytes each)
constexpr int64_t kSmallK = 256;
// Longest thin sector GEMM that joins the tensor-core launch when the contraction has one anyway: a
// few padded tiles there, against a launch of its own (22 to 30 us for the edge charges of a
// chi = 2048 environment, whose 32 x 32 FMAs per row sit on a few SMs).
constexpr int64_t kTiledThin = 4096;

}  // namespace

void plan_direct(const std::vector<MapProblem>& map, const std::vector<GemmTask>& gemms,
                 int num_sms, DirectTables& t) {
  int64_t fma = 0, axes = 0, kmax = 0, thin_rows = 0;
  bool tiled = false;
  for (const MapProblem& q : map) {
    fma += q.M * q.N * std::max<int64_t>(q.K, 1);
    axes += q.M + q.N + q.K;
    kmax = std::max(kmax, q.K);
    if (q.K <= kThinMax && std::min(q.M, q.N) <= kThinMax) thin_rows += std::max(q.M, q.N);
    else tiled = true;
  }
  const bool small = fma <= kSmallFma && axes <= kSmallAxes && kmax <= kSmallK;
  // rows per thin unit: about eight units per SM, so that staging a unit's tables is shared by many rows
  // and the last wave is short (four or two: the chi = 1024 environment 125 -> 136, 155 us)
  const int64_t unit = std::min<int64_t>(
      2048, std::max<int64_t>(256, (thin_rows / (8 * num_sms) + 255) / 256 * 256));
  for (size_t p = 0; p < map.size(); ++p) {
    const MapProblem& q = map[p];
    auto axis = [&](const std::vector<AxisCombo>& c) {
      const int32_t at = (int32_t)t.axes.size();
      append_axis(c, t.axes);
      return at;
    };
    auto table = [&](const std::vector<MapBlock>& b) {
      const int32_t at = (int32_t)t.blocks.size();
      t.blocks.insert(t.blocks.end(), b.begin(), b.end());
      return at;
    };
    if (small) {
      SmallProblem s{};
      s.first = (int32_t)t.small_tiles;
      s.M = (int32_t)q.M;
      s.N = (int32_t)q.N;
      s.K = (int32_t)q.K;
      s.mt = (int32_t)((q.M + kSmallRows - 1) / kSmallRows);
      s.axM = axis(q.m);
      s.axN = axis(q.n);
      s.axK = axis(q.k);
      s.nkc = (int32_t)q.k.size();
      s.nnc = (int32_t)q.n.size();
      s.blkA = table(q.A);
      s.blkB = table(q.B);
      s.blkC = table(q.C);
      t.small_tiles += s.mt * ((q.N + kSmallCols - 1) / kSmallCols);
      t.small.push_back(s);
    } else if (q.K <= kThinMax && std::min(q.M, q.N) <= kThinMax &&
               !(tiled && std::max(q.M, q.N) <= kTiledThin)) {
      const bool longB = q.M < q.N;
      const auto &lc = longB ? q.n : q.m, &tc = longB ? q.m : q.n;
      const auto &tl = longB ? q.B : q.A, &tt = longB ? q.A : q.B;
      std::vector<AxisEntry> te, ke;
      append_axis(tc, te);
      append_axis(q.k, ke);
      auto at = [](const AxisEntry& e, const int32_t* str) {
        int64_t o = 0;
        for (int d = 0; d < kMapLegs; ++d) o += (int64_t)e.i[d] * str[d];
        return o;
      };
      const int32_t vals = (int32_t)t.vals.size();
      for (const AxisEntry& x : te)
        for (const AxisEntry& y : ke) {
          const MapBlock& b = tt[(x.combo_run & kComboMask) * q.k.size() +
                                 (y.combo_run & kComboMask)];
          t.vals.push_back(b.base + at(x, b.rs) + at(y, b.cs));
        }
      for (size_t i = 0; i < lc.size(); ++i) {
        const int32_t offs = (int32_t)t.offs.size();
        for (const AxisEntry& y : ke) {
          const MapBlock& b = tl[i * q.k.size() + (y.combo_run & kComboMask)];
          t.offs.push_back(ThinOffset{b.base + at(y, b.cs), b.rs[0], b.rs[1], b.rs[2], 0});
        }
        for (const AxisEntry& x : te) {
          const size_t j = x.combo_run & kComboMask;
          const MapBlock& b = longB ? q.C[j * lc.size() + i] : q.C[i * tc.size() + j];
          const int32_t *row = longB ? b.cs : b.rs, *thin = longB ? b.rs : b.cs;
          t.offs.push_back(ThinOffset{b.base + at(x, thin), row[0], row[1], row[2], 0});
        }
        for (int64_t r = 0; r < lc[i].count; r += unit) {
          ThinUnit u{};
          u.T = (int32_t)te.size();
          u.K = (int32_t)ke.size();
          u.longB = longB;
          u.offs = offs;
          u.vals = vals;
          u.start = (int32_t)r;
          u.count = (int32_t)std::min<int64_t>(unit, lc[i].count - r);
          u.d0 = (uint32_t)lc[i].d[0];
          u.d1 = (uint32_t)lc[i].d[1];
          magic_u31(u.d0, u.m0, u.s0);
          magic_u31(u.d1, u.m1, u.s1);
          t.units.push_back(u);
        }
      }
    } else {
      t.tiled.push_back(f64tc::Task{gemms[p], &q});
    }
  }
  std::stable_sort(t.units.begin(), t.units.end(),
                   [](const ThinUnit& a, const ThinUnit& b) { return a.count > b.count; });
}

bool DirectPlan::build(const ContractPlan& p, const TensorMeta& A, const TensorMeta& B,
                       int num_sms, cudaStream_t st, bool ca, bool cb) {
  std::vector<MapProblem> map = build_contract_map(p, A, B);
  if (ca || cb) map = complex_map(map, ca, cb);
  if (map.empty()) return false;
  std::vector<GemmTask> gemms = p.mm.gemms;  // (addresses come from the map)
  for (GemmTask& g : gemms) {
    if (ca) g.M *= 2;
    if (cb) g.N *= 2;
  }
  DirectTables t;
  plan_direct(map, gemms, num_sms, t);
  for (const auto& x : t.tiled)
    if (!f64tc::eligible(x.g)) return false;
  // nothing to save: the operands and the result are the fused matrices already
  if (!ca && !cb && !t.tiled.empty() && p.fa.identity && p.fb.identity && p.split.identity) return false;
  stream = st;
  flops = p.flops * (ca ? 2 : 1) * (cb ? 2 : 1);
  for (const auto& x : t.tiled) tc_flops += 2.0 * x.g.M * x.g.N * x.g.K;
  TableImage img;
  const size_t os = img.add(t.small), ou = img.add(t.units), of = img.add(t.offs),
               ov = img.add(t.vals), oa = img.add(t.axes), ob = img.add(t.blocks);
  d_tables = img.upload(st);
  table_bytes = img.bytes.size();
  d_small = (SmallProblem*)(d_tables + os);
  d_units = (ThinUnit*)(d_tables + ou);
  d_offs = (ThinOffset*)(d_tables + of);
  d_vals = (int64_t*)(d_tables + ov);
  d_axes = (AxisEntry*)(d_tables + oa);
  d_blocks = (MapBlock*)(d_tables + ob);
  nsmall = (int)t.small.size();
  nunits = (int)t.units.size();
  small_tiles = (int)t.small_tiles;
  for (const ThinUnit& x : t.units) thin_k = std::max(thin_k, x.K);
  if (!t.tiled.empty()) {
    tc = std::make_unique<f64tc::Plan>();
    tc->build(t.tiled, num_sms, st);
  }
  return true;
}

DirectPlan::~DirectPlan() {
  if (d_tables) cudaFreeAsync(d_tables, stream);
}

// (re, im) of a complex product from its four real ones, with the arithmetic of two linear combinations
// in one pass and launch.
__global__ void __launch_bounds__(256) complex_parts_kernel(int64_t n, double* __restrict__ rr,
                                                            double* __restrict__ ri,
                                                            const double* ir, const double* ii,
                                                            double c_ri, double c_ir, double c_ii) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    rr[e] = fma(c_ii, ii[e], fma(1.0, rr[e], 0.0));
    ri[e] = fma(c_ir, ir[e], fma(c_ri, ri[e], 0.0));
  }
}

void launch_complex_parts(Context* ctx, int64_t n, double* rr, double* ri, const double* ir,
                          const double* ii, double c_ri, double c_ir, double c_ii) {
  if (n == 0) return;
  const int64_t grid = std::min<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8);
  launch_chained(complex_parts_kernel, dim3((unsigned)grid), dim3(256), 0, ctx->stream, 1, n, rr, ri,
                 ir, ii, c_ri, c_ir, c_ii);
  ctx->kernel_launches++;
}

bool launch_direct(Context* ctx, DirectPlan& p, const double* A, const double* B, double* C,
                   const PartOffsets& parts) {
  cudaStream_t st = ctx->stream;
  if (p.tc && !f64tc::launch(ctx, *p.tc, A, B, C, parts)) return false;
  if (p.small_tiles || p.nunits) {
    KernelTimer timer(ctx, kKindGemmF64, p.flops - p.tc_flops);
    if (p.small_tiles) {
      const int grid = std::min(p.small_tiles, ctx->num_sms * 16);
      launch_chained(contract_small_kernel, dim3((unsigned)grid), dim3(kSmallRows * kSmallCols), 0, st,
                     1, p.d_small, p.nsmall, p.small_tiles, p.d_axes, p.d_blocks, A, B, C, parts);
      ctx->kernel_launches++;
    }
    if (p.nunits) {
      // Rows in flight per thread by the longest K. Two for K <= 4: with four (114 registers, two CTAs
      // per SM) a two-site H_eff takes 98 us instead of 90 at chi = 517 and 536 instead of 523 at
      // 2048, with one 540 there.
      auto kern = p.thin_k <= 4   ? contract_thin_kernel<4, 2>
                  : p.thin_k <= 8 ? contract_thin_kernel<8, 2>
                  : p.thin_k <= 16 ? contract_thin_kernel<16, 1>
                                   : contract_thin_kernel<32, 1>;
      const int grid = std::min(p.nunits, ctx->num_sms * 8);
      launch_chained(kern, dim3((unsigned)grid), dim3(256), 0, st, 1, p.d_units, p.nunits, p.d_offs,
                     p.d_vals, A, B, C, parts);
      ctx->kernel_launches++;
    }
  }
  ctx->gemm_flops += p.flops;
  return true;
}

}  // namespace mpsg
