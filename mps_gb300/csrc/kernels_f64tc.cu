// FP64 grouped block GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), FP64 in,
// FP64-accurate out.
//
// GB300 issues 2 FP64 FMAs per SM and clock (1.1 TFLOP/s measured with cuBLAS), so a sector GEMM
// on the FP64 pipe is bound by it from a few blocks on. Here every operand row is written as
// 61-bit fixed point relative to its largest element and cut into seven balanced 9-bit digits,
// each exact in bf16; the digit products run on the tensor cores and are summed exactly:
//
//   * Packing (pack_f64_kernel). For row r of an operand (row of A, column of B) with |x| < 2^e,
//     F = round(x 2^(61-e)) = sum_p t_p 2^(9 (6-p)), |t_0| <= 128, -256 <= t_p <= 255; slice p
//     stores t_p 2^(-9p), which bf16's 8 significant bits hold exactly (|t_p| <= 2^8). The digits
//     are the 9-bit fields of F + 2^8 (1 + 2^9 + ... + 2^45).
//   * MMA. Slice pair (p, q) with p + q <= 6 belongs to group g = p + q, of weight 2^(-9g); 28
//     pairs. Groups 0..4 have a TMEM accumulator each, groups 5 and 6 share one: 6 x 80 = 480 of
//     the 512 columns. One K index adds at most 2^14, 2^16, 2^17, 3 2^16, 2^18 units of 2^(-9g)
//     to groups 0..4, so the FP32 sums over 1024, 256, 128, 64, 64 columns (drain_steps) are exact
//     integers of at most 2^24. The shared accumulator rounds at 2^-24 of a sum of weight 2^-45,
//     far below the last bit of the result.
//   * Drain. After those many columns the epilogue warps add a group's accumulator, groups 0..4
//     as integers into one 64-bit fixed-point sum per output element (unit 2^-36; for K > kWideK
//     unit 2^-27, group 4 joining the small ones) and the small groups into one FP32 sum. At the
//     end both are rounded to FP64 once. No FP64 instruction is issued.
//
// Every operand element is off by at most 2^-62 of its row's largest, products of weight 2^-63 and
// less are left out, and the result is rounded once, where a chain of K FP64 FMAs rounds K times.
//
// A row with a non-finite element, or whose largest element is outside 2^-400..2^400, is marked
// in its exponent; every output element of such a row or column is computed in the epilogue by
// the chain of FP64 FMAs over k, as the FP64-pipe kernel does, so NaN, infinities, overflow and
// subnormals come out as there.
//
// Tile 128 x 80: six accumulators of 80 columns fill TMEM. A K step of 32 is 56 MMAs (about 66 cycles
// each, issue and shared-memory reads of 6.5 KB per MMA) against 91 KB of operands from L2 (about
// 2900 cycles). A group is drained while the others' MMAs run: groups 3 and 4, drained every
// second step, come last within a step, and every accumulator has its own pair of barriers. Tiles are
// cut along K where whole tiles would leave SMs idle (plan_group).
//
// Measured: one 4096 x 4000 x 4096 product 2.72 ms (49 TFLOP/s of FP64 work, 74% of the bf16 rate in
// digit products; the FP64 pipe takes 125 ms). Before the MMAs were issued from code that the
// whole warp runs in step (elect_one) 3.72 ms: 80 cycles per MMA went into moving its operands to
// uniform registers. A two-site H_eff (packing, this kernel, two thin
// steps, packing, this kernel) takes 521 us at chi = 2048 (9680 on the FP64 pipe) and 89 us at chi = 517
// (1005); at chi = 2048 this kernel is 2 x 160 us of it, tensor cycles 42 and 53%: the epilogue's integer
// sums and stores of a tile, 13000 cycles, hold the next one's MMAs up. Relative error of N(0,1)
// products against extended precision: 2e-16 (K = 33) to 1.4e-15 (K = 2050) on the FP64 pipe, 5e-17 here.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "dep_load.cuh"
#include "f64tc.hpp"
#include "tc5.cuh"

namespace mpsg {
namespace f64tc {

using namespace tc;

namespace {

namespace cg = cooperative_groups;

constexpr int kAccs = 6;
constexpr int kBits = 9;                   // per digit
constexpr int64_t kWideK = 8000;           // K 2^14.02 2^36 < 2^63

// K steps between drains of accumulator g (a power of two), and whether step ks of nk begins / ends
// such a stretch.
__device__ __forceinline__ constexpr int drain_steps(int g) {
  return g == 0 || g == kAccs - 1 ? 32 : g == 1 ? 8 : g == 2 ? 4 : 2;
}
__device__ __forceinline__ bool drain_begin(int g, int ks) {
  return (ks & (drain_steps(g) - 1)) == 0;
}
__device__ __forceinline__ bool drain_end(int g, int ks, int nk) {
  return ((ks + 1) & (drain_steps(g) - 1)) == 0 || ks == nk - 1;
}
constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2;
constexpr int kStageBytes = kSlices * (kABytes + kBBytes);  // 91 KB
constexpr int kStages = 2;
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
constexpr int kTmemCols = 512;
constexpr int kEpiWarps = 20;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kEpiCols = BN * 4 / kEpiWarps;  // 16 columns per epilogue thread

constexpr int kRowZero = 1 << 20;  // exponent entry of an all-zero row
constexpr int kRowBad = 1 << 21;   // ... of a row outside the sliced range (see above)
constexpr int kExpRange = 400;
constexpr int kRowBlock = 32;      // rows per packing item

// Adds one accumulator element of an exact group G (v a multiple of 2^(-9G)) into a 64-bit sum in
// units of 2^-U.
template <int G, int U>
__device__ __forceinline__ void add_group(long long& hi, float v) {
  const int i = __float2int_rn(v * __uint_as_float((uint32_t)(127 + kBits * G) << 23));
  hi += (long long)i << (U - kBits * G);
}

// Groups 3 and 4 are drained every second K step. Their MMAs come last in a step, so that the other
// groups' run while they are drained.
__device__ __forceinline__ constexpr bool late_group(int g) { return g == 3 || g == 4; }

// The MMAs of one K step for the early (pass 0) or late (pass 1) groups, slice of R by slice of R:
// consecutive MMAs read that slice from shared memory once (collector hint), which is what bounds
// MMAs of 80 columns otherwise.
__device__ __forceinline__ void issue_pass(int pass, uint32_t tmem, uint32_t sA, uint32_t sB,
                                           int ks) {
  constexpr uint32_t idesc = make_idesc(BM, BN);
#pragma unroll
  for (int pa = 0; pa < kSlices; ++pa) {
    int first = -1, last = -1;  // slices of S that meet slice pa of R in this pass
#pragma unroll
    for (int q = 0; q < kSlices - pa; ++q)
      if (late_group(pa + q) == (pass == 1)) {
        if (first < 0) first = q;
        last = q;
      }
    if (first < 0) continue;
    const uint64_t ad = sw64_desc(sA + pa * kABytes);
#pragma unroll
    for (int kk = 0; kk < BK / 16; ++kk) {
#pragma unroll
      for (int q = 0; q < kSlices - pa; ++q) {
        if (late_group(pa + q) != (pass == 1)) continue;
        const int g = pa + q < kAccs ? pa + q : kAccs - 1;
        const uint32_t d = tmem + (uint32_t)(g * BN);
        const uint64_t a = ad + 2 * kk, b = sw64_desc(sB + q * kBBytes) + 2 * kk;
        // the first MMA of a stretch overwrites the accumulator
        const uint32_t acc =
            pa == 0 && kk == 0 && q <= kAccs - 1 && drain_begin(g, ks) ? 0u : 1u;
        if (first == last) umma_bf16_a<kDiscardA>(d, a, b, idesc, acc);
        else if (q == first) umma_bf16_a<kFillA>(d, a, b, idesc, acc);
        else if (q == last) umma_bf16_a<kLastA>(d, a, b, idesc, acc);
        else umma_bf16_a<kUseA>(d, a, b, idesc, acc);
      }
    }
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Adds 8 columns of one chunk's accumulator g into (hi, lo).
template <bool WIDE>
__device__ __forceinline__ void drain8(uint32_t taddr, int g, long long* hi, float* lo) {
  constexpr int U = WIDE ? 27 : 36;
  uint32_t v[8];
  tmem_ld8(taddr, v);
  tmem_wait();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float x = __uint_as_float(v[j]);
    switch (g) {
      case 0: add_group<0, U>(hi[j], x); break;
      case 1: add_group<1, U>(hi[j], x); break;
      case 2: add_group<2, U>(hi[j], x); break;
      case 3: add_group<3, U>(hi[j], x); break;
      case 4:
        if constexpr (WIDE) lo[j] += x;
        else add_group<4, U>(hi[j], x);
        break;
      default: lo[j] += x;
    }
  }
}

// (hi 2^-U + lo) 2^E rounded to nearest even (integer instructions; the result is in the normal
// range). hi moves up by the free bits it has, at most 24, before lo joins it.
__device__ __forceinline__ double sum_to_f64(long long hi, float lo, int U, int E) {
  const unsigned long long mag = hi < 0 ? 0ull - (unsigned long long)hi : (unsigned long long)hi;
  const int sh = max(0, min(24, __clzll((long long)mag) - 2));
  const long long a = (long long)((unsigned long long)hi << sh) +
                      __float2ll_rn(lo * __uint_as_float((uint32_t)(127 + U + sh) << 23));
  if (a == 0) return 0.0;
  const unsigned long long sign = (unsigned long long)a & (1ull << 63);
  unsigned long long u = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  const int lz = __clzll((long long)u);
  u <<= lz;  // bit 63 set
  // adding the mantissa (without its top bit) to the exponent field lets a carry of the rounding
  // move on into the exponent
  const unsigned long long rest = u & 0x7ffull;
  unsigned long long bits = (u >> 11) & ((1ull << 52) - 1);
  bits += (rest > 0x400ull) || (rest == 0x400ull && (bits & 1ull)) ? 1ull : 0ull;
  bits += (unsigned long long)(63 - lz - U - sh + E + 1023) << 52;
  return __longlong_as_double((long long)(sign | bits));
}

__device__ __forceinline__ AxisEntry load_entry(const AxisEntry* e) {
  const int4 v = __ldg(reinterpret_cast<const int4*>(e));
  return AxisEntry{v.x, {v.y, v.z, v.w}};
}

constexpr int kRun = 8;  // elements that run8 fetches

// How a kernel finds elements: by strides (kFused), through block tables (kMapped), or through block
// tables that name one of several tensors (kParts).
enum Access { kFused, kMapped, kParts };

// Base of a block, with the distance of the part it is in.
template <bool PARTS>
struct PartBase {
  __device__ __forceinline__ PartBase(int64_t, int64_t, int64_t) {}
  __device__ __forceinline__ int64_t of(int64_t base) const { return base; }
};
template <>
struct PartBase<true> {
  int64_t p1, p2, p3;
  __device__ __forceinline__ PartBase(int64_t a, int64_t b, int64_t c) : p1(a), p2(b), p3(c) {}
  __device__ __forceinline__ int64_t of(int64_t base) const { return part_base(base, p1, p2, p3); }
};

// Addresses along one row of an operand or of the output: strided, or through the block table row
// `tab` of the row's combo (a new block is looked up when the column's combo changes).
struct FusedCursor {
  int64_t at0, step;
  __device__ __forceinline__ FusedCursor(const MapBlock*, const AxisEntry*, int64_t o, int64_t row,
                                         int64_t rs, int64_t cs, int64_t, int64_t = 0, int64_t = 0)
      : at0(o + row * rs), step(cs) {}
  __device__ __forceinline__ int64_t at(const AxisEntry*, int64_t col) { return at0 + col * step; }
  // x[j] = X[element col + j], zero from column `end` on
  __device__ __forceinline__ void run8(const double* X, const AxisEntry*, int64_t col, int64_t end,
                                       double (&x)[kRun]) {
    const double* p = X + at0 + col * step;
#pragma unroll
    for (int j = 0; j < kRun; ++j) x[j] = col + j < end ? load_dep(p + j * step) : 0.0;
  }
};

template <bool PARTS>
struct MapCursor {
  const MapBlock* tab;
  AxisEntry r;
  int combo = -1, row = 0, c0 = 0, c1 = 0, c2 = 0;
  int64_t base = 0;
  PartBase<PARTS> parts;
  // tab: the table's first block, ncol blocks per row combo; entry: the row's axis entry; p1..p3:
  // distances of the parts
  __device__ __forceinline__ MapCursor(const MapBlock* t, const AxisEntry* entry, int64_t, int64_t,
                                       int64_t, int64_t ncol, int64_t p1, int64_t p2 = 0,
                                       int64_t p3 = 0)
      : parts(p1, p2, p3) {
    r = load_entry(entry);
    tab = t + (int64_t)(r.combo_run & kComboMask) * ncol;
  }
  __device__ __forceinline__ int64_t at(const AxisEntry* cols, int64_t col) {
    return at(load_entry(cols + col));
  }
  __device__ __forceinline__ int64_t at(const AxisEntry& e) {
    if ((e.combo_run & kComboMask) != combo) {
      combo = e.combo_run & kComboMask;
      const int4* b = reinterpret_cast<const int4*>(tab + combo);
      const int4 x = __ldg(b), y = __ldg(b + 1);
      base = parts.of((int64_t)(((unsigned long long)(unsigned)x.y << 32) | (unsigned)x.x));
      row = r.i[0] * x.z + r.i[1] * x.w + r.i[2] * y.x;
      c0 = y.y;
      c1 = y.z;
      c2 = y.w;
    }
    return base + (row + e.i[0] * c0 + e.i[1] * c1 + e.i[2] * c2);
  }
  __device__ __forceinline__ void run8(const double* X, const AxisEntry* cols, int64_t col,
                                       int64_t end, double (&x)[kRun]) {
    const AxisEntry e = load_entry(cols + col);
    if ((uint32_t)e.combo_run >> 24 >= kRun) {  // one stride (the run ends with the axis at most)
      const double* p = X + at(e);
      const int64_t step = c0;
#pragma unroll
      for (int j = 0; j < kRun; ++j) x[j] = load_dep(p + j * step);
      return;
    }
    int64_t a[kRun];
#pragma unroll
    for (int j = 0; j < kRun; ++j) a[j] = col + j < end ? at(cols, col + j) : 0;
#pragma unroll
    for (int j = 0; j < kRun; ++j) x[j] = col + j < end ? load_dep(X + a[j]) : 0.0;
  }
};

template <Access MAP>
using Cursor = std::conditional_t<MAP == kFused, FusedCursor, MapCursor<MAP == kParts>>;

constexpr int64_t kSlotWords = (int64_t)BM * BN * 2;  // 64-bit words of a cut tile's sums

// One cluster per item (32 rows of one operand, whole K), its K steps shared out over the CTAs: each
// CTA keeps its part in shared memory while it finds the rows' largest elements, the CTAs exchange
// those, and the digits are cut from the kept part. HBM and L2 see 8 bytes read and 14 written
// per element; about 60 integer and FP32 instructions. A part longer than kCacheSteps (K above
// 8 x 192) is read again instead of kept: four CTAs fit an SM so, three with eight steps.
constexpr int kCacheSteps = 6, kPadRows = kRowBlock + 1, kMaxCluster = 8;

template <Access MAP>
__global__ void __launch_bounds__(256) pack_f64_kernel(
    const Problem* __restrict__ probs, const int2* __restrict__ items, int ncta, int cache_steps,
    const AxisEntry* __restrict__ axes, const MapBlock* __restrict__ blocks,
    const double* A, const double* B, int32_t* __restrict__ RA,
    int32_t* __restrict__ RB, __nv_bfloat16* __restrict__ packA, __nv_bfloat16* __restrict__ packB,
    int64_t rowsA, int64_t rowsB, int* __restrict__ arrivals, ulonglong2* __restrict__ slots,
    int nslots, int64_t partA, int64_t partB) {
  extern __shared__ double xs[];  // [k][row], rows padded to kPadRows
  __shared__ uint32_t red[8][33], rlow[8][33];  // largest high words, all low words or-ed
  __shared__ uint2 rmax[kRowBlock];
  __shared__ int rexp[kRowBlock];
  cudaTriggerProgrammaticLaunchCompletion();
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int rank = blockIdx.x % ncta;
  const int2 item = items[blockIdx.x / ncta];
  const int side = (item.x >> 30) & 1;
  const Problem& P = probs[item.x & 0x3fffffff];
  const int64_t r0 = item.y, K = P.K;
  const int64_t rows = side ? P.N : P.M, rs = side ? P.brs : P.ars;
  const int64_t kstep = MAP ? P.nkc : (side ? P.bks : P.aks);
  const double* X = ((P.swap != 0) != (side != 0)) ? B : A;
  const int64_t part = ((P.swap != 0) != (side != 0)) ? partB : partA;
  const int64_t x0 = side ? P.ob : P.oa;
  const MapBlock* tab = blocks + (side ? P.blkB : P.blkA);
  const AxisEntry* row_ax = axes + (side ? P.axN : P.axM);
  const AxisEntry* k_ax = axes + P.axK;
  const int nr = (int)min((int64_t)kRowBlock, rows - r0);
  const int per = (P.nk + ncta - 1) / ncta;
  const int s0 = min(rank * per, P.nk), s1 = min(s0 + per, P.nk);
  const int64_t kb = (int64_t)s0 * BK, ke = min((int64_t)s1 * BK, K);
  const bool keep = per <= cache_steps;
  cudaGridDependencySynchronize();
  // the GEMM's arrival counters and the sums of its cut tiles
  if (blockIdx.x == 0)
    for (int i = t; i < nslots; i += blockDim.x) arrivals[i] = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + t; i < nslots * (kSlotWords / 2);
       i += (int64_t)gridDim.x * blockDim.x)
    slots[i] = make_ulonglong2(0, 0);
  // largest |x| of each row's part: lanes along whichever axis is contiguous
  if (side ? P.fastB : P.fastA) {
    uint32_t m = 0, lo = 0;
    if (lane < nr) {
      Cursor<MAP> c(tab, row_ax + r0 + lane, x0, r0 + lane, rs, kstep, part);
      for (int64_t k = kb + w * kRun; k < (int64_t)s1 * BK; k += 8 * kRun) {
        double x[kRun];
        if (k < ke) {
          c.run8(X, k_ax, k, ke, x);
        } else {
#pragma unroll
          for (int j = 0; j < kRun; ++j) x[j] = 0.0;
        }
        double* keep_at = xs + (int)(k - kb) * kPadRows + lane;
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
          m = max(m, (uint32_t)__double2hiint(x[j]) & 0x7fffffffu);
          lo |= (uint32_t)__double2loint(x[j]);
          if (keep) keep_at[j * kPadRows] = x[j];  // zero beyond K (the part holds whole steps)
        }
      }
    }
    red[w][lane] = m;
    rlow[w][lane] = lo;
  } else {
    for (int rr = w; rr < kRowBlock; rr += 8) {
      uint32_t m = 0, lo = 0;
      if (rr < nr) {
        Cursor<MAP> c(tab, row_ax + r0 + rr, x0, r0 + rr, rs, kstep, part);
#pragma unroll 4
        for (int64_t k = kb + lane; k < ke; k += 32) {
          const double x = load_dep(X + c.at(k_ax, k));
          m = max(m, (uint32_t)__double2hiint(x) & 0x7fffffffu);
          lo |= (uint32_t)__double2loint(x);
          if (keep) xs[(int)(k - kb) * kPadRows + rr] = x;
        }
        if (keep && kb < ke && ke == K)  // zeros up to the whole step
          for (int64_t k = ke + lane; k < (int64_t)s1 * BK; k += 32)
            xs[(int)(k - kb) * kPadRows + rr] = 0.0;
      }
      m = __reduce_max_sync(0xffffffffu, m);
      lo = __reduce_or_sync(0xffffffffu, lo);
      if (lane < 8) {
        red[lane][rr] = m;
        rlow[lane][rr] = lo;
      }
    }
  }
  __syncthreads();
  if (t < kRowBlock) {
    uint32_t m = 0, lo = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      m = max(m, red[g][t]);
      lo |= rlow[g][t];
    }
    rmax[t] = make_uint2(m, lo);
  }
  if (ncta > 1) cg::this_cluster().sync();
  else __syncthreads();
  if (t < kRowBlock) {
    uint2 m = rmax[t];
    for (int q = 1; q < ncta; ++q) {
      const uint2 o = *cg::this_cluster().map_shared_rank(&rmax[t], (rank + q) % ncta);
      m = make_uint2(max(m.x, o.x), m.y | o.y);
    }
    int e = (int)(m.x >> 20) - 1022;  // |x| < 2^e for the row's largest |x|
    if ((m.x | m.y) == 0) e = kRowZero;
    else if (e < -kExpRange || e > kExpRange) e = kRowBad;  // also Inf and NaN
    rexp[t] = e;
    if (rank == 0 && t < nr) (side ? RB + P.rB : RA + P.rA)[r0 + t] = e;
  }
  // no CTA leaves, and none goes on, before the others have read its maxima
  if (ncta > 1) cg::this_cluster().sync();
  else __syncthreads();
  // digits: a warp covers 8 rows x 32 K of one step, a thread 8 consecutive K of a row
  const int rr = (w & 3) * 8 + (lane >> 2), g8 = (lane & 3) * 8;
  if (rr >= nr) return;
  const int rpt = side ? BN : BM;
  const int64_t r = r0 + rr;
  const int64_t tile0 = (side ? P.tB : P.tA) + (r / rpt) * P.nk;
  const int64_t plane = (side ? rowsB : rowsA) * BK;
  __nv_bfloat16* out = (side ? packB : packA) + (r % rpt) * BK + g8;
  const int e = rexp[rr];
  Cursor<MAP> c(tab, row_ax + r, x0, r, rs, kstep, part);
  for (int s = s0 + (w >> 2); s < s1; s += 2) {
    const int64_t k0 = (int64_t)s * BK + g8;
    double x[kRun];
    if (keep) {
      const double* p = xs + (int)(k0 - kb) * kPadRows + rr;
#pragma unroll
      for (int j = 0; j < kRun; ++j) x[j] = p[j * kPadRows];
    } else if (k0 < K) {
      c.run8(X, k_ax, k0, K, x);
    } else {
#pragma unroll
      for (int j = 0; j < kRun; ++j) x[j] = 0.0;
    }
    uint32_t packed[kSlices][4];
    float prev[kSlices];
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
      const uint32_t hw = (uint32_t)__double2hiint(x[j]), lw = (uint32_t)__double2loint(x[j]);
      // |x| 2^(61-e), rounded half up: the 53-bit significand as 62 bits (one below the unit),
      // shifted right by the distance d >= 0 to the row's largest exponent (63: nothing is left,
      // as for zeros, subnormals and every element of a row that is not sliced)
      const int d = min(e + 1022 - (int)((hw >> 20) & 0x7ffu), 63);
      const unsigned long long m9 =
          ((unsigned long long)(((hw & 0xfffffu) | 0x100000u) << 9 | lw >> 23) << 32) | (lw << 9);
      const unsigned long long F = ((m9 >> d) + 1) >> 1;
      const unsigned long long sgn = (unsigned long long)((long long)(int)hw >> 63);
      // 2^8 in every 9-bit field, so that all fields are >= 0
      const unsigned long long G = ((F ^ sgn) - sgn) + 0x4020100804020100ull;
      const uint32_t top = (uint32_t)(G >> 36), mid = (uint32_t)(G >> 9), low = (uint32_t)G;
#pragma unroll
      for (int q = 0; q < kSlices; ++q) {
        // field of digit q as mantissa bits p .. p + 8 of a number of exponent 23 - p - 9q: the
        // number minus 2^(23-p-9q) (1 + 2^(8+p-23)) is the digit times 2^(-9q)
        const uint32_t word = q < 3 ? top : q < 6 ? mid : low;
        const int at = q < 6 ? kBits * (2 - q % 3) : 0, p = at > 14 ? 0 : at;
        const uint32_t f = at > 14 ? (word >> at) & 0x1ffu : word & (0x1ffu << p);
        const uint32_t magic = (uint32_t)(150 - p - kBits * q) << 23;
        const float v = __uint_as_float(f | magic) - __uint_as_float(magic | (256u << p));
        if (j & 1) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(prev[q], v);  // exact
          packed[q][j >> 1] = *reinterpret_cast<const uint32_t*>(&h);
        } else {
          prev[q] = v;
        }
      }
    }
    const int64_t idx = (tile0 + s) * rpt * BK;
#pragma unroll
    for (int q = 0; q < kSlices; ++q)
      *reinterpret_cast<uint4*>(out + q * plane + idx) =
          make_uint4(packed[q][0], packed[q][1], packed[q][2], packed[q][3]);
  }
}

// Output elements n0 .. n0 + nc of one row that are not sliced (the row, or the element's column, is
// marked): the chain of FP64 FMAs over k.
template <Access MAP>
__device__ __noinline__ void fma_chains(const Problem& P, int64_t row, int64_t n0, int nc,
                                        bool all, const int32_t* RB, const AxisEntry* axes,
                                        const MapBlock* blocks, const double* R, const double* S,
                                        double* C, const PartOffsets& parts) {
  const AxisEntry *m_ax = axes + P.axM + row, *n_ax = axes + P.axN, *k_ax = axes + P.axK;
  Cursor<MAP> out(blocks + P.blkC, m_ax, P.oc, row, P.crs, MAP ? P.nnc : P.ccs,
                  parts.c1, parts.c2, parts.c3);
  for (int j = 0; j < nc; ++j) {
    if (!all && RB[j] != kRowBad) continue;
    Cursor<MAP> a(blocks + P.blkA, m_ax, P.oa, row, P.ars, MAP ? P.nkc : P.aks,
                  P.swap ? parts.b : parts.a);
    Cursor<MAP> b(blocks + P.blkB, n_ax + n0 + j, P.ob, n0 + j, P.brs, MAP ? P.nkc : P.bks,
                  P.swap ? parts.a : parts.b);
    double y = 0.0;
    for (int64_t k = 0; k < P.K; ++k) y = fma(R[a.at(k_ax, k)], S[b.at(k_ax, k)], y);
    C[out.at(n_ax, n0 + j)] = y;
  }
}


// Persistent, one CTA per SM: warp 0 TMA producer, warp 1 TMEM allocator and MMA issuer, 20
// epilogue warps (five per TMEM lane quarter, 16 columns each). Every mbarrier wait is bounded;
// on expiry the kernel records an error code, stops issuing, waits for its own MMAs and frees
// TMEM.
template <Access MAP>
__global__ void __launch_bounds__(kThreads, 1) gemm_f64tc_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
    const Problem* __restrict__ probs, const Tile* __restrict__ tiles, int64_t ntiles,
    const int32_t* RA, const int32_t* RB,
    const AxisEntry* __restrict__ axes, const MapBlock* __restrict__ blocks,
    const double* A, const double* B, double* __restrict__ C,
    unsigned long long* __restrict__ slots, int* __restrict__ arrivals, int* __restrict__ err,
    const __grid_constant__ PartOffsets parts) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + kStages * kStageBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kStages;
  uint64_t* tfull = bars + 2 * kStages;  // one pair per accumulator
  uint64_t* tempty = tfull + kAccs;
  uint64_t* esync = tempty + kAccs;  // all epilogue threads
  uint64_t* drain = esync + 1;
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile int* last_part = (volatile int*)(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int g = 0; g < kAccs; ++g) {
      mbar_init(&tfull[g], 1);
      mbar_init(&tempty[g], 32 * kEpiWarps);
    }
    mbar_init(esync, 32 * kEpiWarps);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      fence_proxy_async_global();
      int stage = 0;
      uint32_t phase = 0;
      for (int64_t i = 0; !*abort_flag; ++i) {
        const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
        if (pos >= ntiles) break;
        const Tile tr = tiles[pos];
        const int nk = probs[tr.prob].nk;
        const int rowA = (int)((probs[tr.prob].tA + (int64_t)tr.mi * nk) * BM);
        const int rowB = (int)((probs[tr.prob].tB + (int64_t)tr.ni * nk) * BN);
        for (int ks = tr.ks0; ks < tr.ks1; ++ks) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, err, 1)) break;
          uint8_t* sA = smem + stage * kStageBytes;
          uint8_t* sB = sA + kSlices * kABytes;
          mbar_expect_tx(&full[stage], kStageBytes);
#pragma unroll
          for (int s = 0; s < kSlices; ++s) {
            tma_load_3d(sA + s * kABytes, &tmA, &full[stage], 0, rowA + ks * BM, s);
            tma_load_3d(sB + s * kBBytes, &tmB, &full[stage], 0, rowB + ks * BN, s);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the warp in step, one lane issues) ----------------
    const uint32_t tmem = warp_uniform(tmem_base);
    int stage = 0;
    uint32_t phase = 0, uses = 0;  // uses: parity of each accumulator's stretches
    bool issued = false, ok = true;
    for (int64_t i = 0; ok; ++i) {
      const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
      if (pos >= ntiles) break;
      const int nk = (int)warp_uniform((uint32_t)(tiles[pos].ks1 - tiles[pos].ks0));
      for (int ks = 0; ks < nk; ++ks) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, err, 3));
        if (!ok) break;
        tc_fence_after();
        const uint32_t sA = warp_uniform(smem_u32(smem + stage * kStageBytes));
        const uint32_t sB = sA + kSlices * kABytes;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
          for (int g = kAccs - 1; g >= 0; --g)
            if (late_group(g) == (pass == 1) && drain_begin(g, ks) && ok) {
              // the accumulator's last stretch has been drained
              ok = __all_sync(0xffffffffu, mbar_wait(&tempty[g], ((uses >> g) & 1) ^ 1,
                                                     abort_flag, err, 2));
              tc_fence_after();
            }
          if (!ok) break;
          issued = true;
          if (elect_one()) {
            issue_pass(pass, tmem, sA, sB, ks);
#pragma unroll
            for (int g = kAccs - 1; g >= 0; --g)
              if (late_group(g) == (pass == 1) && drain_end(g, ks, nk)) umma_commit(&tfull[g]);
            if (pass == 1) umma_commit(&empty[stage]);
          }
          __syncwarp();
#pragma unroll
          for (int g = kAccs - 1; g >= 0; --g)
            if (late_group(g) == (pass == 1) && drain_end(g, ks, nk)) uses ^= 1u << g;
        }
        if (!ok) break;
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (issued) {  // make sure every MMA has retired before TMEM is released
      if (elect_one()) umma_commit(drain);
      __syncwarp();
      volatile int no_abort = 0;
      mbar_wait(drain, 0, &no_abort, err, 4);
    }
  } else {
    // ---------------- epilogue ----------------
    const int lrow = 32 * (warp & 3) + lane;  // TMEM lane = tile row
    const int col0 = ((warp - 2) >> 2) * kEpiCols;
    const uint32_t taddr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
    uint32_t uses = 0;
    for (int64_t i = 0;; ++i) {
      const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
      if (pos >= ntiles) break;
      const Tile tr = tiles[pos];
      const Problem& P = probs[tr.prob];
      const int nk = tr.ks1 - tr.ks0;
      const int64_t K = P.K;
      const bool wide = K > kWideK;
      long long hi[kEpiCols];
      float lo[kEpiCols];
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j) {
        hi[j] = 0;
        lo[j] = 0.f;
      }
      bool ok = true;
      for (int ks = 0; ks < nk && ok; ++ks) {
#pragma unroll
        for (int i = 0; i < kAccs; ++i) {
          // the order of their commits: 5, 2, 1, 0, then 4, 3
          const int g = i == 0 ? kAccs - 1 : i < 4 ? 3 - i : 8 - i;
          if (!drain_end(g, ks, nk)) continue;
          ok = ok && mbar_wait(&tfull[g], (uses >> g) & 1, abort_flag, err, 5);
          if (!ok) break;
          uses ^= 1u << g;
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < kEpiCols; h += 8) {
            if (wide) drain8<true>(taddr + g * BN + h, g, hi + h, lo + h);
            else drain8<false>(taddr + g * BN + h, g, hi + h, lo + h);
          }
          tc_fence_before();
          mbar_arrive(&tempty[g]);
        }
      }
      if (!ok) break;
      const int64_t row = (int64_t)tr.mi * BM + lrow, n0 = (int64_t)tr.ni * BN + col0;
      const int nc = (int)min((int64_t)kEpiCols, P.N - n0);
      if (tr.parts > 1) {
        // element (row, column) at column * BM + row of the tile's slot: the 64-bit sums, then the small
        // ones in units of 2^-60 (integers both, so their order does not matter)
        unsigned long long* s = slots + tr.slot * kSlotWords + col0 * BM + lrow;
        if (row < P.M) {
#pragma unroll
          for (int j = 0; j < kEpiCols; ++j)
            if (j < nc) {
              atomicAdd(s + j * BM, (unsigned long long)hi[j]);
              atomicAdd(s + BM * BN + j * BM,
                        (unsigned long long)__float2ll_rn(lo[j] * __uint_as_float((127u + 60u) << 23)));
            }
        }
        __threadfence();
        mbar_arrive(esync);  // every thread's sums are on their way before the arrival counts
        if (!mbar_wait(esync, 0, abort_flag, err, 6)) break;
        if (threadIdx.x == 64) {
          __threadfence();
          *last_part = atomicAdd(arrivals + tr.slot, 1) == tr.parts - 1;
        }
        mbar_arrive(esync);
        if (!mbar_wait(esync, 1, abort_flag, err, 6)) break;
        if (!*last_part) continue;
        __threadfence();
        if (row < P.M) {
#pragma unroll
          for (int j = 0; j < kEpiCols; ++j) {
            hi[j] = j < nc ? (long long)__ldcg(s + j * BM) : 0;
            const long long l = j < nc ? (long long)__ldcg(s + BM * BN + j * BM) : 0;
            lo[j] = (float)l * __uint_as_float((127u - 60u) << 23);
          }
        }
      }
      if (row < P.M) {
        const int er = K ? RA[P.rA + row] : kRowZero;
        const int32_t* RBp = RB + P.rB + n0;
        bool bad = er == kRowBad;
#pragma unroll
        for (int j = 0; j < kEpiCols; ++j) {  // the sums' registers take the FP64 bits
          const int ec = K && j < nc ? RBp[j] : kRowZero;
          bad = bad || ec == kRowBad;
          const double y = er >= kRowZero || ec >= kRowZero
                               ? 0.0
                               : sum_to_f64(hi[j], lo[j], wide ? 27 : 36, er + ec - 14);
          hi[j] = __double_as_longlong(y);
        }
        Cursor<MAP> out(blocks + P.blkC, axes + P.axM + row, P.oc, row, P.crs,
                        MAP ? P.nnc : P.ccs, parts.c1, parts.c2, parts.c3);
        const AxisEntry* n_ax = axes + P.axN;
#pragma unroll
        for (int j = 0; j < kEpiCols; ++j) {
          if (j >= nc) break;
          C[out.at(n_ax, n0 + j)] = __longlong_as_double(hi[j]);
        }
        if (bad)
          fma_chains<MAP>(P, row, n0, nc, er == kRowBad, RBp, axes, blocks, P.swap ? B : A,
                          P.swap ? A : B, C, parts);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

constexpr size_t kGroupBytes = size_t(2) << 30;  // packed operands per launch pair
// Pieces of a tile. They may be as short as one K step: with three as the least, the chi = 363 right
// environment takes 68.3 us instead of 65.8, a chi = 256 eigensolve 2.04 ms instead of 2.00.
constexpr int kMaxParts = 16;
// (with 1.5 for kCutSteps chi = 2048 takes 562 us instead of 549, chi = 517 the same)
constexpr double kCutSteps = 2.5, kTileSteps = 1.0;

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

size_t packed_bytes(const GemmTask& t) {
  return (size_t)(ceil_div(t.M, BM) * BM + ceil_div(t.N, BN) * BN + 128) *
         (size_t)(ceil_div(t.K, BK) * BK) * 2 * kSlices;
}

}  // namespace

// Every tiled task (K > 32, or M and N > 32) is faster here, down to the smallest: a 64 x 64 tile
// takes the FP64 pipe 2048 cycles per k index, whatever part of it is padding, and the tensor
// cores about 120 (chi = 48: 55 us a GEMM against 21 with its packing). Beyond kMaxK the
// 64-bit sums could overflow; such a K is left to the FP64 pipe.
bool eligible(const GemmTask& t) { return t.K <= kMaxK; }

size_t Group::scratch_bytes() const {
  return round256((size_t)rowsA * BK * 2 * kSlices) + round256((size_t)rowsB * BK * 2 * kSlices) +
         round256(sizeof(int32_t) * (size_t)rA) + round256(sizeof(int32_t) * (size_t)rB) +
         round256(sizeof(int) * (size_t)nslots) + (size_t)nslots * kSlotWords * 8;
}

// Whether the rows of an operand table, rather than k, run along the unit stride of its blocks
// (judged on its largest block).
static bool rows_fast(const std::vector<MapBlock>& tab, const std::vector<AxisCombo>& rows,
                      const std::vector<AxisCombo>& k) {
  size_t i = 0, j = 0;
  for (size_t x = 0; x < rows.size(); ++x)
    if (rows[x].count > rows[i].count) i = x;
  for (size_t x = 0; x < k.size(); ++x)
    if (k[x].count > k[j].count) j = x;
  const MapBlock& b = tab[i * k.size() + j];
  int32_t best_r = 0, best_k = 0;  // longest unit-stride run on either side
  for (int d = 0; d < kMapLegs; ++d) {
    if (b.rs[d] == 1) best_r = std::max(best_r, rows[i].d[d]);
    if (b.cs[d] == 1) best_k = std::max(best_k, k[j].d[d]);
  }
  return best_r >= best_k;
}

void plan_group(const std::vector<Task>& g, int num_sms, Group& G, GroupTables& t) {
  int64_t tA = 0, tB = 0, rA = 0, rB = 0;
  G.flops = 0;
  for (const Task& task : g) {
    const GemmTask& x = task.g;
    Problem P{};
    // The operand whose rows run along the unit stride of the output takes the 128-row side, so that an
    // epilogue warp stores whole lines (8 bytes of each otherwise: two-site H_eff, chi = 2048 581 us instead of 557),
    // unless the other way round pads at least a fifth fewer tiles.
    const int64_t direct = ceil_div(x.M, BM) * ceil_div(x.N, BN);
    const int64_t swapped = ceil_div(x.N, BM) * ceil_div(x.M, BN);
    const bool rows = !task.map || rows_fast(task.map->C, task.map->m, task.map->n);
    P.swap = rows ? 5 * swapped < 4 * direct : 4 * swapped <= 5 * direct;
    P.K = x.K;
    P.oc = x.offC;
    if (!P.swap) {
      P.M = x.M;
      P.N = x.N;
      P.oa = x.offA;
      P.ars = 1;
      P.aks = x.lda;
      P.ob = x.offB;
      P.brs = x.ldb;
      P.bks = 1;
      P.crs = 1;
      P.ccs = x.ldc;
    } else {
      P.M = x.N;
      P.N = x.M;
      P.oa = x.offB;
      P.ars = x.ldb;
      P.aks = 1;
      P.ob = x.offA;
      P.brs = 1;
      P.bks = x.lda;
      P.crs = x.ldc;
      P.ccs = 1;
    }
    P.fastA = P.ars == 1;
    P.fastB = P.brs == 1;
    P.mt = (int32_t)ceil_div(P.M, BM);
    P.nt = (int32_t)ceil_div(P.N, BN);
    P.nk = (int32_t)ceil_div(P.K, BK);
    P.tA = tA;
    P.tB = tB;
    P.rA = rA;
    P.rB = rB;
    tA += (int64_t)P.mt * P.nk;
    tB += (int64_t)P.nt * P.nk;
    rA += P.M;
    rB += P.N;
    if (const MapProblem* q = task.map) {
      const auto &rm = P.swap ? q->n : q->m, &rn = P.swap ? q->m : q->n;
      const auto &ta = P.swap ? q->B : q->A, &tb = P.swap ? q->A : q->B;
      P.axM = (int32_t)t.axes.size();
      append_axis(rm, t.axes);
      P.axN = (int32_t)t.axes.size();
      append_axis(rn, t.axes);
      P.axK = (int32_t)t.axes.size();
      append_axis(q->k, t.axes);
      P.nkc = (int32_t)q->k.size();
      P.nnc = (int32_t)rn.size();
      P.blkA = (int32_t)t.blocks.size();
      t.blocks.insert(t.blocks.end(), ta.begin(), ta.end());
      P.blkB = (int32_t)t.blocks.size();
      t.blocks.insert(t.blocks.end(), tb.begin(), tb.end());
      P.blkC = (int32_t)t.blocks.size();
      for (size_t i = 0; i < rm.size(); ++i)
        for (size_t j = 0; j < rn.size(); ++j) {
          MapBlock b = P.swap ? q->C[j * rm.size() + i] : q->C[i * rn.size() + j];
          if (P.swap) std::swap(b.rs, b.cs);
          t.blocks.push_back(b);
        }
      if (P.K > 0) {
        P.fastA = rows_fast(ta, rm, q->k);
        P.fastB = rows_fast(tb, rn, q->k);
      }
    }
    const int p = (int)t.probs.size();
    for (int ni = 0; ni < P.nt; ++ni)
      for (int mi = 0; mi < P.mt; ++mi) t.tiles.push_back(Tile{p, mi, ni, 0, P.nk, 0, 0, 1});
    if (P.K > 0) {
      for (int64_t r = 0; r < P.M; r += kRowBlock) t.items.push_back(make_int2(p, (int)r));
      for (int64_t r = 0; r < P.N; r += kRowBlock)
        t.items.push_back(make_int2(p | (1 << 30), (int)r));
    }
    G.flops += 2.0 * x.M * x.N * x.K;
    G.tasks.push_back(x);
    t.probs.push_back(P);
  }
  // Tiles of very different K, or fewer tiles than SMs, leave SMs idle: then tiles are cut along K
  // into pieces of at most `most` K steps, which add their sums up in L2. A piece costs that (160 KB,
  // and for the last one its way back; about kCutSteps K steps), a tile its first loads and its stores
  // (kTileSteps); the limit with the shortest estimated busiest SM is taken, the uncut list first.
  auto cut_at = [&](int most, std::vector<Tile>& cut, int64_t& slots) {
    cut.clear();
    slots = 0;
    for (const Tile& x : t.tiles) {
      const int parts = std::min<int>(kMaxParts, (int)ceil_div(std::max(x.ks1, 1), most));
      for (int q = 0; q < parts; ++q) {
        Tile y = x;
        y.ks0 = (int)((int64_t)x.ks1 * q / parts);
        y.ks1 = (int)((int64_t)x.ks1 * (q + 1) / parts);
        y.slot = (int32_t)slots;
        y.part = q;
        y.parts = parts;
        cut.push_back(y);
      }
      if (parts > 1) ++slots;
    }
    std::stable_sort(cut.begin(), cut.end(), [](const Tile& a, const Tile& b) {
      return a.ks1 - a.ks0 > b.ks1 - b.ks0;
    });
    const int64_t sms = std::min<int64_t>(num_sms, (int64_t)cut.size());
    std::vector<double> load((size_t)std::max<int64_t>(sms, 1), 0.0);
    for (int64_t i = 0; i < (int64_t)cut.size(); ++i) {
      const int64_t r = i / sms, c = i % sms;  // the kernel's snake order
      load[(size_t)((r & 1) ? sms - 1 - c : c)] +=
          cut[i].ks1 - cut[i].ks0 + kTileSteps + (cut[i].parts > 1 ? kCutSteps : 0.0);
    }
    return *std::max_element(load.begin(), load.end());
  };
  std::vector<Tile> cut, best;
  int64_t slots = 0, max_nk = 1;
  for (const Tile& x : t.tiles) max_nk = std::max<int64_t>(max_nk, x.ks1);
  double span = cut_at((int)max_nk, best, G.nslots), even = 0.0;
  for (const Tile& x : best) even += (x.ks1 - x.ks0 + kTileSteps) / num_sms;
  for (int d = 2; d <= kMaxParts && d <= max_nk && span > 1.1 * even; ++d) {
    const double s = cut_at((int)ceil_div(max_nk, d), cut, slots);
    if (s < 0.95 * span) {
      span = s;
      best = cut;
      G.nslots = slots;
    }
  }
  cut = std::move(best);
  t.tiles = std::move(cut);
  std::stable_sort(t.items.begin(), t.items.end(), [&](const int2& a, const int2& b) {
    return t.probs[a.x & 0x3fffffff].K > t.probs[b.x & 0x3fffffff].K;
  });
  G.nprob = (int)t.probs.size();
  G.ntiles = (int64_t)t.tiles.size();
  G.nitems = (int)t.items.size();
  for (const Problem& P : t.probs) G.max_nk = std::max(G.max_nk, P.nk);
  G.rowsA = std::max<int64_t>(tA, 1) * BM;
  G.rowsB = std::max<int64_t>(tB, 1) * BN;
  G.rA = rA;
  G.rB = rB;
}

void Plan::build(const std::vector<Task>& g, int num_sms, cudaStream_t st) {
  release();
  stream = st;
  mapped = !g.empty() && g[0].map != nullptr;
  std::vector<std::vector<Task>> parts;
  size_t bytes = 0;
  for (const Task& t : g) {
    const size_t b = packed_bytes(t.g);
    if (parts.empty() || (bytes > 0 && bytes + b > kGroupBytes)) {
      parts.emplace_back();
      bytes = 0;
    }
    parts.back().push_back(t);
    bytes += b;
  }
  for (const auto& part : parts) {
    groups.emplace_back();
    Group& G = groups.back();
    GroupTables t;
    plan_group(part, num_sms, G, t);
    TableImage img;
    const size_t op = img.add(t.probs), ot = img.add(t.tiles), oi = img.add(t.items),
                 oa = img.add(t.axes), ob = img.add(t.blocks);
    G.d_tables = img.upload(st);
    G.d_probs = (Problem*)(G.d_tables + op);
    G.d_tiles = (Tile*)(G.d_tables + ot);
    G.d_items = (int2*)(G.d_tables + oi);
    G.d_axes = (AxisEntry*)(G.d_tables + oa);
    G.d_blocks = (MapBlock*)(G.d_tables + ob);
  }
}

double Plan::flops() const {
  double f = 0;
  for (const Group& G : groups) f += G.flops;
  return f;
}

void Plan::release() {
  for (Group& G : groups) {
    if (G.d_tables) cudaFreeAsync(G.d_tables, stream);
    if (G.plain) G.plain->release();
  }
  groups.clear();
}

template <Access MAP>
static void launch_group(Context* ctx, Group& G, unsigned char* mem, const double* A,
                         const double* B, double* C, const PartOffsets& parts) {
  static std::once_flag smem_set[kMaxDevices], pack_set[kMaxDevices];
  cudaStream_t st = ctx->stream;
  const size_t bA = round256((size_t)G.rowsA * BK * 2 * kSlices),
               bB = round256((size_t)G.rowsB * BK * 2 * kSlices);
  __nv_bfloat16* packA = (__nv_bfloat16*)mem;
  __nv_bfloat16* packB = (__nv_bfloat16*)(mem + bA);
  int32_t* RA = (int32_t*)(mem + bA + bB);
  int32_t* RB = (int32_t*)(mem + bA + bB + round256(sizeof(int32_t) * (size_t)G.rA));
  int* arrivals = (int*)((unsigned char*)RB + round256(sizeof(int32_t) * (size_t)G.rB));
  unsigned long long* slots =
      (unsigned long long*)((unsigned char*)arrivals + round256(sizeof(int) * (size_t)G.nslots));
  CUtensorMap tmA, tmB;
  make_slice_map(&tmA, packA, G.rowsA, kSlices, BM, BK, BK);
  make_slice_map(&tmB, packB, G.rowsB, kSlices, BN, BK, BK);
  set_smem_limit_once(ctx, smem_set, gemm_f64tc_kernel<MAP>, kSmemBytes);
  if (G.nitems) {
    KernelTimer timer(ctx, kKindPack);
    // CTAs per item: as many as keep an item's part in shared memory, and more while that fills the chip
    // (up to eight CTAs per SM, a CTA's barriers and latencies being most of its time; two K steps
    // each are worth one). Two-site H_eff, one CTA per eight steps / so: chi = 517 106 / 98 us, 2048
    // 550 / 536; complex one-site product 122 / 111 us. With four steps as the limit, or more CTAs
    // than that, chi = 2048 and 1024 lose what the small ones gain.
    int ncta = 1;
    while (ncta < kMaxCluster &&
           (ceil_div(G.max_nk, ncta) > kCacheSteps ||
            (ceil_div(G.max_nk, ncta) > 2 && G.nitems * ncta * 2 <= 8 * ctx->num_sms)))
      ncta *= 2;
    const int steps = (int)std::min<int64_t>(kCacheSteps, ceil_div(G.max_nk, ncta));
    const int smem = steps * BK * kPadRows * (int)sizeof(double);
    set_smem_limit_once(ctx, pack_set, pack_f64_kernel<MAP>,
                        kCacheSteps * BK * kPadRows * (int)sizeof(double));
    launch_chained(pack_f64_kernel<MAP>, dim3((unsigned)G.nitems * (unsigned)ncta), dim3(256),
                   (size_t)smem, st, ncta, G.d_probs, G.d_items, ncta, steps, G.d_axes, G.d_blocks,
                   A, B, RA, RB, packA, packB, G.rowsA, G.rowsB, arrivals, (ulonglong2*)slots,
                   (int)G.nslots, parts.a,
                   parts.b);
    ctx->kernel_launches++;
  }
  KernelTimer timer(ctx, kKindGemmF64, G.flops);
  const int grid = (int)std::min<int64_t>(G.ntiles, ctx->num_sms);
  launch_chained(gemm_f64tc_kernel<MAP>, dim3((unsigned)grid), dim3(kThreads), (size_t)kSmemBytes, st,
                 1, tmA, tmB, G.d_probs, G.d_tiles, G.ntiles, RA, RB, G.d_axes, G.d_blocks, A, B, C,
                 slots, arrivals, ctx->wait_err + kWaitGemm, parts);
  ctx->kernel_launches++;
}

bool launch(Context* ctx, Plan& p, const double* A, const double* B, double* C,
            const PartOffsets& parts) {
  cudaStream_t st = ctx->stream;
  for (Group& G : p.groups) {
    if (G.ntiles == 0) continue;
    unsigned char* mem = nullptr;
    const cudaError_t e = cudaMallocAsync((void**)&mem, G.scratch_bytes(), st);
    if (e == cudaErrorMemoryAllocation) {
      // no room for the packed operands (twice the FP64 ones): the FP64-pipe kernel needs none
      (void)cudaGetLastError();
      if (p.mapped) return false;
      if (!G.plain) {
        G.plain = std::make_unique<DevGemmPlan>();
        G.plain->upload(G.tasks, G.flops, st);
      }
      launch_gemm_f64(ctx, *G.plain, A, B, C);
      ctx->gemm_flops -= G.flops;  // counted by the caller
      continue;
    }
    MPSG_CUDA(e);
    if (!p.mapped) launch_group<kFused>(ctx, G, mem, A, B, C, parts);
    else if (parts.c1 == 0) launch_group<kMapped>(ctx, G, mem, A, B, C, parts);
    else launch_group<kParts>(ctx, G, mem, A, B, C, parts);
    MPSG_CUDA(cudaFreeAsync(mem, st));
  }
  if (ctx->debug_sync) {
    MPSG_CUDA(cudaStreamSynchronize(st));
    check_waits(ctx);
  }
  return true;
}

}  // namespace f64tc
}  // namespace mpsg
