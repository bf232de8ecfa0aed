// FP64 grouped block GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), FP64 in,
// FP64-accurate out.
//
// GB300 issues 2 FP64 FMAs per SM and clock (1.1 TFLOP/s measured with cuBLAS), so a sector GEMM
// on the FP64 pipe is bound by it from a few blocks on. Here every operand row is written as
// 79-bit fixed point relative to its largest element and cut into nine balanced 9-bit digits,
// each exact in bf16; the digit products run on the tensor cores and are summed exactly:
//
//   * Packing (pack_f64_kernel). For row r of an operand (row of A, column of B) with |x| < 2^e,
//     F = floor(x 2^(79-e)) = sum_p t_p 2^(9 (8-p)), |t_0| <= 128, -256 <= t_p <= 255; slice p
//     stores t_p 2^(-9p), which bf16's 8 significant bits hold exactly (|t_p| <= 2^8). The digits
//     are the 9-bit fields of F + 2^8 (1 + 2^9 + ... + 2^72).
//   * MMA. Slice pair (p, q) belongs to group g = p + q, of weight 2^(-9g). A tile takes the pairs of
//     its mode: 28 (g <= 6, the first seven digits), 34 (g <= 7) or all 45 (g <= 8). Every group has
//     a TMEM accumulator of 64 columns, but the last two share one, in the first and the last mode.
//     One K index adds at most 2^14, 2^16, 2^17, 3 2^16, 2^18, 5 2^16, 6 2^16 units of 2^(-9g) to groups
//     0..6, so the FP32 sums over 1024, 256, 128, 64, 64, 32, 32 columns (drain_steps) are exact integers
//     of at most 2^24. What rounds (a shared accumulator; groups 5 and up where not all digits are taken)
//     does so at 2^-24 of a sum of weight 2^-45 at most, below what the mode leaves out.
//   * Drain. After those many columns the epilogue warps add a group's accumulator, groups 0..4
//     as integers into one 64-bit fixed-point sum per output element (unit 2^-36, whole K up to
//     kWideK; longer K is cut into pieces) and the others into a second one (unit 2^-63, or FP32).
//     At the end both are rounded to FP64 once. No FP64 instruction is issued.
//
// Accuracy, element by element, however the operands are graded (mode_of): what is left out is below 2^-53
// of sum |a b| rms, or below what a chain of K FP64 FMAs rounds rms, and at most K 2^-51 of sum |a b|; an
// element for which that cannot be shown is computed by FP64 FMAs (fma_element). For operands of one size the
// result is rounded once, where the chain rounds K times: relative error of N(0,1) products against
// extended precision 2e-16 (K = 33) to 1.4e-15 (K = 2050) on the FP64 pipe, 5e-17 here.
//
// A row with a non-finite element, or whose largest element is outside 2^-400..2^400, is marked
// in its exponent; every output element of such a row or column is computed in the epilogue by
// the chain of FP64 FMAs over k, as the FP64-pipe kernel does, so NaN, infinities, overflow and
// subnormals come out as there.
//
// Tile 128 x 64: eight accumulators of 64 columns fill TMEM. A K step of 32 is 56, 68 or 90 MMAs (about
// 55 to 66 cycles each) against 86 or 108 KB of operands from L2. A group is drained while the others'
// MMAs run: those drained every step or every second one come last within a step, and every
// accumulator has its own pair of barriers. Tiles are cut along K where whole tiles would leave SMs
// idle (plan_group).
//
// Measured: one 4096 x 4000 x 4096 product 3.3 ms (40 TFLOP/s of FP64 work; the FP64 pipe takes 125 ms).
// Before the MMAs were issued from code that the whole warp runs in step (elect_one) they took 80 cycles
// each, most of them to move their operands to uniform registers. A two-site H_eff (packing, this
// kernel, two thin steps, packing, this kernel) takes 574 us at chi = 2048 (9680 on the FP64 pipe) and
// 96 us at chi = 517 (1005). Seven digits and no bound for the elements, as 128 x 80 tiles, took 522 and 90
// us, and lost all digits of a small element next to a large one. The same with every element of the
// tensors scaled by a power of ten of its own, over 3, 8, 16 decades: 774, 782, 827 us at chi = 2048,
// 113, 115, 162 at chi = 517.
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

constexpr int kAccs = 8;                   // accumulators, at most
constexpr int kBits = 9;                   // per digit
constexpr int64_t kWideK = 8000;           // K 2^14.02 2^36 < 2^63; longer K is cut into pieces
constexpr int kWideSteps = (int)(kWideK / BK);

// How many digit products a tile takes (see tile_mode): those of seven digits with p + q <= 6, with
// p + q <= 7, or those of all nine with p + q <= 8.
enum Mode { kFew = 0, kMore = 1, kAll = 2 };
template <int MODE>
struct Digits {
  static constexpr int n = MODE == kAll ? kSlices : kFewSlices;
  static constexpr int groups = 7 + MODE;
  // one per group, but the last two of kFew (5, 6) and of kAll (7, 8) share one
  static constexpr int accs = MODE == kFew ? 6 : kAccs;
};

// K steps between drains of accumulator g (a power of two), and whether step ks of nk begins / ends
// such a stretch.
template <int MODE>
__device__ __forceinline__ constexpr int drain_steps(int g) {
  return g == 0 ? 32 : g == 1 ? 8 : g == 2 ? 4 : g <= 4 ? 2 : MODE != kAll ? 32 : 1;
}
template <int MODE>
__device__ __forceinline__ bool drain_begin(int g, int ks) {
  return (ks & (drain_steps<MODE>(g) - 1)) == 0;
}
template <int MODE>
__device__ __forceinline__ bool drain_end(int g, int ks, int nk) {
  return ((ks + 1) & (drain_steps<MODE>(g) - 1)) == 0 || ks == nk - 1;
}
constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2;
constexpr int kStageBytes = kSlices * (kABytes + kBBytes);  // 108 KB
constexpr int kStages = 2;
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256 + BM * BN / 8;  // (barriers, words: 224)
constexpr int kTmemCols = 512;
static_assert(kAccs * BN <= kTmemCols, "accumulators fit TMEM");
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kEpiCols = BN * 4 / kEpiWarps;  // 16 columns per epilogue thread
static_assert(kEpiWarps == 16 && kEpiCols == 16, "finish_tile shares out columns modulo 16");

constexpr int kExpRange = 400;
// A row's entry: its exponent << kCountBits | its number of middling elements (see mode_of), K at most.
constexpr int kCountBits = 17, kCountMask = (1 << kCountBits) - 1;
constexpr int kRowZero = 1000;  // exponent of an all-zero row
constexpr int kRowBad = 1001;   // ... of a row outside the sliced range (see above)
static_assert(kMaxK <= kCountMask && kExpRange < kRowZero, "counts and exponents fit an entry");
constexpr int kRowBlock = 32;      // rows per packing item
static_assert(BM % kRowBlock == 0 && BN % kRowBlock == 0, "a row block is in one tile");

// Which digit products. A row's bound is the power of two above its largest element, RR the product of a
// row's and a column's; an element is large from 2^-kLargeBits of its row's bound on. la and lb are the
// smallest numbers of large elements of a row in the tile's row blocks of either operand: any row and column
// have n = la + lb - K of them at the same k at least, so S = sum |a b| >= n 2^-10 RR. Left out are
//   kFew   sqrt(K) 2^-61.3 RR rms, at most K 2^-58.4 RR (the products of weight 2^-63),
//   kMore  sqrt(K) 2^-65.6 RR rms, at most K 2^-61 RR (the rounding of the elements),
// each taken where that is below 2^-53 S rms and, at worst, below the worst case of the FMA chain,
// K 2^-53 S. kAll leaves out sqrt(K) 2^-79 RR rms, K 2^-75 RR at most. The FMA chain's rounding is about
// 0.4 sqrt(K) 2^-53 S rms where the terms have one sign and 2^-54.5 S where the signs are random, |y| being
// about S and S / sqrt(K) then: in both cases no less than kAll's at |y| = 2^-kGuardBits RR. Smaller outputs are
// computed again by FP64 FMAs, unless their row and column have n >= sqrt(K / 2) elements from 2^-kMidBits of
// their bounds on at the same k (counted likewise; S >= n 2^-24 RR).
// N(0,1) operands pass the first from K of about 60 on, and so does the MPO-contracted intermediate of an XXZ
// H_eff, a sixth of it zeros: 97% of the work at chi = 517, 99% at chi = 1024; the last contraction of
// environment updates 91% and, all but edge charges, the second. Real states are graded: 9 in 10 tiles of a
// chi = 2048 sweep's environments take all digits, and 1.6 million of their 1.2e9 elements FMAs (16
// million with 2^-20 for the guard and no count of middling elements; the sweep's FP64 products take 197 ms
// so, 757 then, 120 with no FMAs, 93 with seven digits and no bound).
constexpr int kLargeBits = 5;
constexpr int kMidBits = 12;
constexpr int kGuardBits = 24;

__device__ __forceinline__ int mode_of(int la, int lb, int64_t K) {
  const int64_t n = (int64_t)la + lb - K;
  if (n < 4 || 36 * n * n < K) return kAll;          // n >= 0.165 sqrt(K)
  return n >= 25 && 2 * n * n >= 21 * K ? kFew : kMore;  // n >= 3.24 sqrt(K)
}

// This lane's count of a tile, and what the warp's say (lanes 0..3 hold R's, 4..7 S's).
__device__ __forceinline__ int tile_count(const Tile& t, const int32_t* LA, const int32_t* LB,
                                          int lane) {
  return lane < t.nA ? LA[t.lA + lane] : lane >= 4 && lane - 4 < t.nB ? LB[t.lB + lane - 4] : t.K;
}
__device__ __forceinline__ int tile_mode(const Tile& t, int count, int lane) {
  const int la = __reduce_min_sync(0xffffffffu, lane < 4 ? count : t.K);
  const int lb = __reduce_min_sync(0xffffffffu, lane < 4 ? t.K : count);
  return mode_of(la, lb, t.K);
}
static_assert(BM / kRowBlock <= 4 && BN / kRowBlock <= 4, "a tile's counts fit the lanes");

// Groups that are drained every step or every second one. Their MMAs come last in a step, so that the
// other groups' run while they are drained.
template <int MODE>
__device__ __forceinline__ constexpr bool late_group(int g) {
  return g == 3 || g == 4 || (MODE == kAll && (g == 5 || g == 6));
}

// The MMAs of one K step for the early (pass 0) or late (pass 1) groups, slice of R by slice of R:
// consecutive MMAs read that slice from shared memory once (collector hint).
template <int MODE>
__device__ __forceinline__ void issue_pass(int pass, uint32_t tmem, uint32_t sA, uint32_t sB,
                                           int ks) {
  constexpr uint32_t idesc = make_idesc(BM, BN);
  constexpr int n = Digits<MODE>::n, groups = Digits<MODE>::groups, accs = Digits<MODE>::accs;
#pragma unroll
  for (int pa = 0; pa < n; ++pa) {
    const int nq = n < groups - pa ? n : groups - pa;
    int first = -1, last = -1;  // slices of S that meet slice pa of R in this pass
#pragma unroll
    for (int q = 0; q < nq; ++q)
      if (late_group<MODE>(pa + q) == (pass == 1)) {
        if (first < 0) first = q;
        last = q;
      }
    if (first < 0) continue;
    const uint64_t ad = sw64_desc(sA + pa * kABytes);
#pragma unroll
    for (int kk = 0; kk < BK / 16; ++kk) {
#pragma unroll
      for (int q = 0; q < nq; ++q) {
        if (late_group<MODE>(pa + q) != (pass == 1)) continue;
        const int g = pa + q < accs ? pa + q : accs - 1;
        const uint32_t d = tmem + (uint32_t)(g * BN);
        const uint64_t a = ad + 2 * kk, b = sw64_desc(sB + q * kBBytes) + 2 * kk;
        // the first MMA of a stretch overwrites the accumulator
        const uint32_t acc =
            pa == (g < n ? 0 : g - n + 1) && kk == 0 && pa + q < accs && drain_begin<MODE>(g, ks) ? 0u
                                                                                                 : 1u;
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

// The sums of an output element: groups 0..4 in units of 2^-kHiUnit, the others of 2^-kLoUnit, or as
// FP32 where all digits are not taken (they are below 2^-27 of the first's unit there, and a 64-bit sum
// would cost the epilogue 16 registers more than it has).
constexpr int kHiUnit = kBits * 4, kLoUnit = kBits * 7;
// A K that is cut because it is long carries kWideShift bits from the first sum into the second.
constexpr int kWideShift = 9;

__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// Adds 8 columns of accumulator g, multiples of 2^(-9g), into (hi, lo).
template <class Lo>
__device__ __forceinline__ void drain8(uint32_t taddr, int g, long long* hi, Lo* lo) {
  uint32_t v[8];
  tmem_ld8(taddr, v);
  tmem_wait();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float x = __uint_as_float(v[j]);
    if (g <= 4) hi[j] += (long long)__float2int_rn(x * pow2f(kBits * g)) << (g <= 4 ? kHiUnit - kBits * g : 0);
    else if constexpr (std::is_same_v<Lo, float>) lo[j] += x;
    else lo[j] += (long long)__float2int_rn(x * pow2f(kBits * g)) << (g > 4 ? kLoUnit - kBits * g : 0);
  }
}

// A second sum in units of 2^-kLoUnit, and back.
__device__ __forceinline__ long long lo_units(float lo) { return __float2ll_rn(lo * pow2f(kLoUnit)); }
__device__ __forceinline__ long long lo_units(long long lo) { return lo; }
__device__ __forceinline__ void lo_from(float& lo, long long l) { lo = (float)l * pow2f(-kLoUnit); }
__device__ __forceinline__ void lo_from(long long& lo, long long l) { lo = l; }
// ... in units of 2^-unit, unit <= kLoUnit
__device__ __forceinline__ long long lo_round(float lo, int unit) { return __float2ll_rn(lo * pow2f(unit)); }
__device__ __forceinline__ long long lo_round(long long lo, int unit) {
  const int down = kLoUnit - unit;
  return down ? ((lo >> (down - 1)) + 1) >> 1 : lo;
}

// (hi 2^-U + lo) 2^E rounded to nearest even (integer instructions; the result is in the normal range).
// hi moves up by the free bits it has, at most to lo's unit, before the upper bits of lo join it.
template <class Lo>
__device__ __forceinline__ double sum_to_f64(long long hi, Lo lo, int U, int E) {
  const unsigned long long mag = hi < 0 ? 0ull - (unsigned long long)hi : (unsigned long long)hi;
  const int sh = max(0, min(kLoUnit - U, __clzll((long long)mag) - 2));
  const long long a = (long long)((unsigned long long)hi << sh) + lo_round(lo, U + sh);
  const unsigned long long sign = (unsigned long long)a & (1ull << 63);
  unsigned long long u = a < 0 ? 0ull - (unsigned long long)a : (unsigned long long)a;
  if (a == 0) return 0.0;
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

constexpr int kRun = 8;  // elements that a thread fetches at once

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
  template <int N>
  __device__ __forceinline__ void run(const double* X, const AxisEntry*, int64_t col, int64_t end,
                                      double (&x)[N]) {
    const double* p = X + at0 + col * step;
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = col + j < end ? load_dep(p + j * step) : 0.0;
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
  template <int N>
  __device__ __forceinline__ void run(const double* X, const AxisEntry* cols, int64_t col,
                                      int64_t end, double (&x)[N]) {
    const AxisEntry e = load_entry(cols + col);
    if ((uint32_t)e.combo_run >> 24 >= N) {  // one stride (the run ends with the axis at most)
      const double* p = X + at(e);
      const int64_t step = c0;
#pragma unroll
      for (int j = 0; j < N; ++j) x[j] = load_dep(p + j * step);
      return;
    }
    int64_t a[N];
#pragma unroll
    for (int j = 0; j < N; ++j) a[j] = col + j < end ? at(cols, col + j) : 0;
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = col + j < end ? load_dep(X + a[j]) : 0.0;
  }
};

template <Access MAP>
using Cursor = std::conditional_t<MAP == kFused, FusedCursor, MapCursor<MAP == kParts>>;

constexpr int64_t kSlotWords = (int64_t)BM * BN * 2;  // 64-bit words of a cut tile's sums

// One cluster per item (32 rows of one operand, whole K), its K steps shared out over the CTAs: each
// CTA keeps its part in shared memory while it finds the rows' largest elements, the CTAs exchange
// those, the digits are cut from the kept part and the large elements of each row counted. HBM and L2 see 8
// bytes read and 18 written per element; about 60 integer and FP32 instructions. A part longer than kCacheSteps (K above
// 8 x 192) is read again instead of kept: four CTAs fit an SM so (three with eight steps, or more than
// 64 registers, which cost the chi = 1024 environment 8% of its packing).
constexpr int kCacheSteps = 6, kPadRows = kRowBlock + 1, kMaxCluster = 8;

template <Access MAP>
__global__ void __launch_bounds__(256, 4) pack_f64_kernel(
    const Problem* __restrict__ probs, const int2* __restrict__ items, int ncta, int cache_steps,
    const AxisEntry* __restrict__ axes, const MapBlock* __restrict__ blocks,
    const double* A, const double* B, int32_t* __restrict__ RA, int32_t* __restrict__ RB,
    int32_t* __restrict__ LA, int32_t* __restrict__ LB, __nv_bfloat16* __restrict__ packA,
    __nv_bfloat16* __restrict__ packB,
    int64_t rowsA, int64_t rowsB, int* __restrict__ arrivals, ulonglong2* __restrict__ slots,
    int nslots, int64_t partA, int64_t partB) {
  extern __shared__ double xs[];  // [k][row], rows padded to kPadRows
  __shared__ uint32_t red[8][33], rlow[8][33];  // largest high words, all low words or-ed
  __shared__ uint2 rmax[kRowBlock];
  __shared__ int rexp[kRowBlock], large[kRowBlock], mid[kRowBlock];  // mode_of's counts
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
          c.run(X, k_ax, k, ke, x);
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
    large[t] = mid[t] = 0;
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
  }
  __syncthreads();
  // digits: a warp covers 4 rows x 32 K of one step, a thread 4 consecutive K of a row (with 8 it takes
  // 80 registers, three CTAs per SM instead of four)
  constexpr int kPer = 4;
  const int rr = w * 4 + (lane & 3), g4 = (lane >> 2) * kPer;  // (no bank conflicts so)
  const int e = rexp[rr] < kRowZero ? rexp[rr] : 1 << 20;
  int counts = 0;  // large elements | middling ones << 16 (of 8 threads: at most 8192)
  if (rr < nr) {
    const int rpt = side ? BN : BM;
    const int64_t r = r0 + rr;
    const int64_t tile0 = (side ? P.tB : P.tA) + (r / rpt) * P.nk;
    const int64_t plane = (side ? rowsB : rowsA) * BK;
    __nv_bfloat16* out = (side ? packB : packA) + (r % rpt) * BK + g4;
    Cursor<MAP> c(tab, row_ax + r, x0, r, rs, kstep, part);
    for (int s = s0; s < s1; ++s) {
      const int64_t k0 = (int64_t)s * BK + g4;
      double x[kPer];
      if (keep) {
        const double* p = xs + (int)(k0 - kb) * kPadRows + rr;
#pragma unroll
        for (int j = 0; j < kPer; ++j) x[j] = p[j * kPadRows];
      } else if (k0 < K) {
        c.run(X, k_ax, k0, K, x);
      } else {
#pragma unroll
        for (int j = 0; j < kPer; ++j) x[j] = 0.0;
      }
      uint32_t packed[kSlices][kPer / 2];
      float prev[kSlices];
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const uint32_t hw = (uint32_t)__double2hiint(x[j]), lw = (uint32_t)__double2loint(x[j]);
        // F = x 2^(79-e) rounded down: M 2^(15-d) in three words, M the 53-bit significand with its top bit
        // at 63 and d >= 0 the distance to the row's largest exponent (nothing is left of zeros,
        // subnormals and the elements of a row that is not sliced), and its complement if x < 0
        const int d = e + 1022 - (int)((hw >> 20) & 0x7ffu);
        counts += (d < kLargeBits) + ((d < kMidBits) << 16);
        const uint32_t m1 = __funnelshift_l(lw, hw, 11) | 0x80000000u, m0 = lw << 11;
        uint32_t f0, f1, f2;
        if (d < 16) {
          f0 = m0 << (15 - d);
          f1 = __funnelshift_l(m0, m1, 15 - d);
          f2 = __funnelshift_l(m1, 0, 15 - d);
        } else {
          const unsigned long long f =
              d > 78 ? 0ull : ((unsigned long long)m1 << 32 | m0) >> (d - 15);
          f0 = (uint32_t)f;
          f1 = (uint32_t)(f >> 32);
          f2 = 0;
        }
        const uint32_t sgn = (uint32_t)((int)hw >> 31);
        // + 2^8 in every 9-bit field, so that all nine fields are >= 0
        f0 ^= sgn;
        f1 ^= sgn;
        f2 ^= sgn;
        asm("add.cc.u32 %0, %0, 0x04020100;\n\taddc.cc.u32 %1, %1, 0x40201008;\n\t"
            "addc.u32 %2, %2, 0x00010080;"
            : "+r"(f0), "+r"(f1), "+r"(f2));
        const uint32_t top = __funnelshift_r(f1, f2, 22), mid = __funnelshift_r(f0, f1, 27), low = f0;
#pragma unroll
        for (int q = 0; q < kSlices; ++q) {
          // field of digit q as mantissa bits p .. p + 8 of a number of exponent 23 - p - 9q: the
          // number minus 2^(23-p-9q) (1 + 2^(8+p-23)) is the digit times 2^(-9q)
          const uint32_t word = q < 3 ? top : q < 6 ? mid : low;
          const int at = kBits * (2 - q % 3), p = at > 14 ? 0 : at;
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
        *reinterpret_cast<uint2*>(out + q * plane + idx) = make_uint2(packed[q][0], packed[q][1]);
    }
  }
  // the fewest large elements of a row, over the rows that the digits stand for
  for (int o = 4; o < 32; o <<= 1) counts += __shfl_xor_sync(0xffffffffu, counts, o);
  if (lane < 4 && counts) {
    const auto cl = cg::this_cluster();
    atomicAdd(ncta > 1 ? cl.map_shared_rank(&large[rr], 0) : &large[rr], counts & 0xffff);
    atomicAdd(ncta > 1 ? cl.map_shared_rank(&mid[rr], 0) : &mid[rr], counts >> 16);
  }
  // (nor does a CTA leave before the others have read its maxima)
  if (ncta > 1) cg::this_cluster().sync();
  else __syncthreads();
  if (rank == 0 && w == 0) {
    const bool sliced = lane < nr && rexp[lane] < kRowZero;
    const int least = __reduce_min_sync(0xffffffffu, sliced ? large[lane] : (int)K);
    if (lane == 0) (side ? LB + P.lB : LA + P.lA)[r0 / kRowBlock] = least;
    if (lane < nr)
      (side ? RB + P.rB : RA + P.rA)[r0 + lane] = rexp[lane] * (kCountMask + 1) + (sliced ? mid[lane] : 0);
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
    if (!all && RB[j] >> kCountBits != kRowBad) continue;
    Cursor<MAP> a(blocks + P.blkA, m_ax, P.oa, row, P.ars, MAP ? P.nkc : P.aks,
                  P.swap ? parts.b : parts.a);
    Cursor<MAP> b(blocks + P.blkB, n_ax + n0 + j, P.ob, n0 + j, P.brs, MAP ? P.nkc : P.bks,
                  P.swap ? parts.a : parts.b);
    double y = 0.0;
    for (int64_t k = 0; k < P.K; ++k) y = fma(R[a.at(k_ax, k)], S[b.at(k_ax, k)], y);
    C[out.at(n_ax, n0 + j)] = y;
  }
}

// Output element (row, col) as FP64 FMAs by a whole warp, a 32nd of k per lane.
template <Access MAP>
__device__ __noinline__ void fma_element(const Problem& P, int64_t row, int64_t col,
                                         const AxisEntry* axes, const MapBlock* blocks,
                                         const double* R, const double* S, double* C,
                                         const PartOffsets& parts) {
  const AxisEntry *m_ax = axes + P.axM + row, *n_ax = axes + P.axN, *k_ax = axes + P.axK;
  const int lane = threadIdx.x & 31;
  Cursor<MAP> a(blocks + P.blkA, m_ax, P.oa, row, P.ars, MAP ? P.nkc : P.aks,
                P.swap ? parts.b : parts.a);
  Cursor<MAP> b(blocks + P.blkB, n_ax + col, P.ob, col, P.brs, MAP ? P.nkc : P.bks,
                P.swap ? parts.a : parts.b);
  double y = 0.0;
#pragma unroll 4
  for (int64_t k = lane; k < P.K; k += 32)
    y = fma(load_dep(R + a.at(k_ax, k)), load_dep(S + b.at(k_ax, k)), y);
  for (int o = 16; o; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
  if (lane == 0) {
    Cursor<MAP> out(blocks + P.blkC, m_ax, P.oc, row, P.crs, MAP ? P.nnc : P.ccs, parts.c1,
                    parts.c2, parts.c3);
    C[out.at(n_ax, col)] = y;
  }
}

// Where a role is in the ring of stages.
struct Ring {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++stage == kStages) {
      stage = 0;
      phase ^= 1;
    }
  }
};

// The MMAs of a tile's nk K steps; false (in all lanes) when a wait has expired. aside(ks) runs after those
// of step ks are issued.
template <int MODE, class Aside>
__device__ __forceinline__ bool mma_tile(int nk, uint32_t tmem, uint8_t* smem, Ring& ring,
                                         uint64_t* full, uint64_t* empty, uint64_t* tfull,
                                         uint64_t* tempty, uint32_t& uses, bool& issued,
                                         volatile int* abort_flag, int* err, const Aside& aside) {
  for (int ks = 0; ks < nk; ++ks) {
    if (!__all_sync(0xffffffffu, mbar_wait(&full[ring.stage], ring.phase, abort_flag, err, 3)))
      return false;
    tc_fence_after();
    const uint32_t sA = warp_uniform(smem_u32(smem + ring.stage * kStageBytes));
    const uint32_t sB = sA + kSlices * kABytes;
    issued = true;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
      for (int g = Digits<MODE>::accs - 1; g >= 0; --g)
        if (late_group<MODE>(g) == (pass == 1) && drain_begin<MODE>(g, ks)) {
          // the accumulator's last stretch has been drained
          if (!__all_sync(0xffffffffu,
                          mbar_wait(&tempty[g], ((uses >> g) & 1) ^ 1, abort_flag, err, 2)))
            return false;
          tc_fence_after();
        }
      if (elect_one()) {
        issue_pass<MODE>(pass, tmem, sA, sB, ks);
#pragma unroll
        for (int g = Digits<MODE>::accs - 1; g >= 0; --g)
          if (late_group<MODE>(g) == (pass == 1) && drain_end<MODE>(g, ks, nk))
            umma_commit(&tfull[g]);
        if (pass == 1) umma_commit(&empty[ring.stage]);
      }
      __syncwarp();
#pragma unroll
      for (int g = Digits<MODE>::accs - 1; g >= 0; --g)
        if (late_group<MODE>(g) == (pass == 1) && drain_end<MODE>(g, ks, nk)) uses ^= 1u << g;
    }
    ring.next();
    aside(ks);
  }
  return true;
}

// What a tile's K steps complete, added to the sums, in the order of the commits; false (in all lanes)
// when a wait has expired.
template <int MODE, class Lo>
__device__ __forceinline__ bool drain_tile(int nk, uint32_t taddr, uint64_t* tfull, uint64_t* tempty,
                                           uint32_t& uses, long long (&hi)[kEpiCols],
                                           Lo (&lo)[kEpiCols], volatile int* abort_flag, int* err) {
  for (int ks = 0; ks < nk; ++ks)
#pragma unroll
    for (int pass = 0; pass < 2; ++pass)
#pragma unroll
      for (int g = Digits<MODE>::accs - 1; g >= 0; --g) {
        if (late_group<MODE>(g) != (pass == 1) || !drain_end<MODE>(g, ks, nk)) continue;
        if (!__all_sync(0xffffffffu, mbar_wait(&tfull[g], (uses >> g) & 1, abort_flag, err, 5)))
          return false;
        uses ^= 1u << g;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < kEpiCols; h += 8) drain8(taddr + g * BN + h, g, hi + h, lo + h);
        tc_fence_before();
        mbar_arrive(&tempty[g]);
      }
  return true;
}

constexpr int kRedoAt = 10;

// What the epilogue of a tile works with.
struct Epilogue {
  uint64_t *tfull, *tempty, *esync;
  volatile int *abort_flag, *last_part;
  const AxisEntry* axes;
  const MapBlock* blocks;
  const int32_t *RA, *RB;
  const double *A, *B;
  double* C;
  unsigned long long* slots;
  int *arrivals, *err;
  uint32_t tmem;  // of this CTA
};

// A tile's epilogue: drains, the sums of a cut tile, rounding and stores. uses: see the caller. False (in all
// lanes) when a wait has expired. ALL: the tile takes all digits.
template <Access MAP, bool ALL>
__device__ __forceinline__ bool finish_tile(const Epilogue& e, const Tile& tr, const Problem& P, int nk,
                                            int mode, uint32_t& uses, const PartOffsets& parts) {
  using Lo = std::conditional_t<ALL, long long, float>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lrow = 32 * (warp & 3) + lane;  // TMEM lane = tile row
  const int col0 = ((warp - 2) >> 2) * kEpiCols;
  const uint32_t taddr = e.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
  const int K = tr.K;
  const bool wide = K > kWideK;
  long long hi[kEpiCols];
  Lo lo[kEpiCols];
#pragma unroll
  for (int j = 0; j < kEpiCols; ++j) {
    hi[j] = 0;
    lo[j] = 0;
  }
  bool ok;
  if constexpr (ALL) {
    ok = drain_tile<kAll>(nk, taddr, e.tfull, e.tempty, uses, hi, lo, e.abort_flag, e.err);
  } else {
    ok = mode == kFew
             ? drain_tile<kFew>(nk, taddr, e.tfull, e.tempty, uses, hi, lo, e.abort_flag, e.err)
             : drain_tile<kMore>(nk, taddr, e.tfull, e.tempty, uses, hi, lo, e.abort_flag, e.err);
  }
  if (!ok) return false;
  const int64_t row = (int64_t)tr.mi * BM + lrow, n0 = (int64_t)tr.ni * BN + col0;
  const int nc = (int)min((int64_t)kEpiCols, P.N - n0);
  if (tr.parts > 1) {
    // element (row, column) at column * BM + row of the tile's slot: the first sums, then the second
    // ones (integers both, so their order does not matter)
    unsigned long long* s = e.slots + tr.slot * kSlotWords + col0 * BM + lrow;
    if (row < P.M) {
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j)
        if (j < nc) {
          long long l = lo_units(lo[j]);
          if (wide) {
            l += (hi[j] & ((1 << kWideShift) - 1)) << (kLoUnit - kHiUnit);
            hi[j] >>= kWideShift;
          }
          atomicAdd(s + j * BM, (unsigned long long)hi[j]);
          atomicAdd(s + BM * BN + j * BM, (unsigned long long)l);
        }
    }
    __threadfence();
    mbar_arrive(e.esync);  // every thread's sums are on their way before the arrival counts
    if (!__all_sync(0xffffffffu, mbar_wait(e.esync, 0, e.abort_flag, e.err, 6))) return false;
    if (threadIdx.x == 64) {
      __threadfence();
      *e.last_part = atomicAdd(e.arrivals + tr.slot, 1) == tr.parts - 1;
    }
    mbar_arrive(e.esync);
    if (!__all_sync(0xffffffffu, mbar_wait(e.esync, 1, e.abort_flag, e.err, 6))) return false;
    if (!*e.last_part) return true;
    __threadfence();
    if (row < P.M) {
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j) {
        hi[j] = j < nc ? (long long)__ldcg(s + j * BM) : 0;
        lo_from(lo[j], j < nc ? (long long)__ldcg(s + BM * BN + j * BM) : 0);
      }
    }
  }
  const double *R = P.swap ? e.B : e.A, *S = P.swap ? e.A : e.B;
  uint32_t redo = 0;  // columns of this row that are left to FMAs
  if (row < P.M) {
    const int ra = K ? e.RA[P.rA + row] : kRowZero << kCountBits, er = ra >> kCountBits;
    const int32_t* RBp = e.RB + P.rB + n0;
    bool bad = er == kRowBad;
#pragma unroll
    for (int j = 0; j < kEpiCols; ++j) {  // the sums' registers take the FP64 bits
      const int rb = K && j < nc ? RBp[j] : kRowZero << kCountBits, ec = rb >> kCountBits;
      bad = bad || ec == kRowBad;
      const double y =
          er >= kRowZero || ec >= kRowZero
              ? 0.0
              : sum_to_f64(hi[j], lo[j], wide ? kHiUnit - kWideShift : kHiUnit, er + ec - 14);
      hi[j] = __double_as_longlong(y);
      if constexpr (ALL) {  // |y| < 2^(er + ec - kGuardBits), by the high word, and too few middling terms
        const int limit = (er + ec - kGuardBits + 1023) << 20;
        const int n = (ra & kCountMask) + (rb & kCountMask) - K;
        if (er < kRowZero && ec < kRowZero && (__double2hiint(y) & 0x7fffffff) < limit &&
            (n < 1 || 2 * (int64_t)n * n < K))
          redo |= 1u << j;
      }
    }
    Cursor<MAP> out(e.blocks + P.blkC, e.axes + P.axM + row, P.oc, row, P.crs, MAP ? P.nnc : P.ccs,
                    parts.c1, parts.c2, parts.c3);
    const AxisEntry* n_ax = e.axes + P.axN;
#pragma unroll
    for (int j = 0; j < kEpiCols; ++j) {
      if (j >= nc) break;
      e.C[out.at(n_ax, n0 + j)] = __longlong_as_double(hi[j]);
    }
    if (bad)
      fma_chains<MAP>(P, row, n0, nc, er == kRowBad, RBp, e.axes, e.blocks, R, S, e.C, parts);
  }
  if constexpr (ALL) {
    // The elements left to FMAs are often those of a few rows or columns: every warp takes those of one
    // diagonal, modulo 16 (with its own rows and columns for each warp, the FP64 products of a chi = 2048
    // sweep's environments and energies take 294 ms instead of 197).
    volatile uint16_t* bits = (volatile uint16_t*)(e.last_part + kRedoAt);  // [tile row][16 columns]
    bits[lrow * 4 + (col0 >> 4)] = (uint16_t)redo;
    mbar_arrive(e.esync);
    if (!__all_sync(0xffffffffu, mbar_wait(e.esync, 0, e.abort_flag, e.err, 6))) return false;
    const int rows = (int)min((int64_t)BM, P.M - (int64_t)tr.mi * BM);
    for (int r0 = 0; r0 < rows; r0 += 32) {  // a row per lane, then the rows that have such elements
      const int r = r0 + lane, c = (warp - 2 + r) & 15;
      uint32_t which = 0;
#pragma unroll
      for (int j = 0; j < BN / 16; ++j)
        which |= (uint32_t)(r < rows ? bits[r * 4 + j] >> c & 1 : 0) << j;
      for (uint32_t todo = __ballot_sync(0xffffffffu, which != 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        for (uint32_t q = __shfl_sync(0xffffffffu, which, l); q; q &= q - 1)
          fma_element<MAP>(P, (int64_t)tr.mi * BM + r0 + l,
                           (int64_t)tr.ni * BN + 16 * (__ffs(q) - 1) + ((warp - 2 + r0 + l) & 15), e.axes,
                           e.blocks, R, S, e.C, parts);
      }
    }
    mbar_arrive(e.esync);  // the next such tile writes the masks again
    if (!__all_sync(0xffffffffu, mbar_wait(e.esync, 1, e.abort_flag, e.err, 6))) return false;
  }
  return true;
}

// The same for all digits, in registers of its own.
template <Access MAP>
__device__ __noinline__ uint2 finish_tile_all(Epilogue e, const Tile* tile, const Problem* P, int nk,
                                              uint32_t uses, PartOffsets parts) {
  const Tile tr = *tile;
  const bool ok = finish_tile<MAP, true>(e, tr, *P, nk, kAll, uses, parts);
  return make_uint2(ok ? 1u : 0u, uses);
}

// Persistent, one CTA per SM: warp 0 TMA producer, warp 1 TMEM allocator and MMA issuer, 16
// epilogue warps (four per TMEM lane quarter, 16 columns each). Every mbarrier wait is bounded;
// on expiry the kernel records an error code, stops issuing, waits for its own MMAs and frees
// TMEM.
template <Access MAP>
__global__ void __launch_bounds__(kThreads, 1) gemm_f64tc_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
    const Problem* __restrict__ probs, const Tile* __restrict__ tiles, int64_t ntiles,
    int64_t ntiles_k, const int32_t* RA, const int32_t* RB, const int32_t* LA, const int32_t* LB,
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
  // What the MMA warp tells the epilogue of tile number i, in word i % kInfo: i << 16 | mode << 13 |
  // K steps. It is at most two tiles ahead, as it waits for the accumulators of the one before.
  constexpr int kInfo = 4;
  volatile uint32_t* info = tmem_slot + 3;
  // ... and after it, kRedoAt words from last_part on, a bit per output element (finish_tile)

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
    for (int q = 0; q < kInfo; ++q) info[q] = ~0u;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  const Tile first = warp < 2 && blockIdx.x < ntiles_k ? tiles[blockIdx.x] : Tile{};
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
      Ring ring;
      for (int64_t i = 0; !*abort_flag; ++i) {
        const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
        if (pos >= ntiles_k) break;
        const Tile tr = i ? tiles[pos] : first;
        int digits = kFewSlices;
        for (int ks = tr.ks0; ks < tr.ks1; ++ks) {
          if (!mbar_wait(&empty[ring.stage], ring.phase ^ 1, abort_flag, err, 1)) break;
          uint8_t* sA = smem + ring.stage * kStageBytes;
          uint8_t* sB = sA + kSlices * kABytes;
          uint64_t* bar = &full[ring.stage];
          auto load = [&](int from, int to) {
            mbar_expect_more(bar, (uint32_t)((to - from) * (kABytes + kBBytes)));
#pragma unroll 1
            for (int s = from; s < to; ++s) {
              tma_load_3d(sA + s * kABytes, &tmA, bar, 0, tr.rowA + ks * BM, s);
              tma_load_3d(sB + s * kBBytes, &tmB, bar, 0, tr.rowB + ks * BN, s);
            }
          };
          load(0, kFewSlices);
          if (ks == tr.ks0) {  // which digits the tile takes is found while the first are on their way
            int la = tr.K, lb = tr.K;
            for (int q = 0; q < tr.nA; ++q) la = min(la, LA[tr.lA + q]);
            for (int q = 0; q < tr.nB; ++q) lb = min(lb, LB[tr.lB + q]);
            if (mode_of(la, lb, tr.K) == kAll) digits = kSlices;
          }
          if (digits > kFewSlices) load(kFewSlices, digits);
          mbar_arrive(bar);
          ring.next();
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the warp in step, one lane issues) ----------------
    const uint32_t tmem = warp_uniform(tmem_base);
    Ring ring;
    uint32_t uses = 0;  // parity of each accumulator's stretches
    bool issued = false, ok = true;
    // the next tile and its counts are fetched while this one's first steps run
    int64_t pos = blockIdx.x;
    Tile next = first;
    int count = pos < ntiles_k ? tile_count(next, LA, LB, lane) : 0;
    for (int64_t i = 0; ok && pos < ntiles_k; ++i) {
      const int nk = (int)warp_uniform((uint32_t)(next.ks1 - next.ks0));
      const int mode = (int)warp_uniform((uint32_t)tile_mode(next, count, lane));
      if (lane == 0)
        info[i % kInfo] = (uint32_t)(i & 0xffff) << 16 | (uint32_t)mode << 13 | (uint32_t)nk;
      pos = sched_pos(i + 1, gridDim.x, blockIdx.x);
      const bool more = pos < ntiles_k;
      auto fetch = [&](int ks) {
        if (ks == 0 && more) next = tiles[pos];
        if (ks == min(1, nk - 1) && more) count = tile_count(next, LA, LB, lane);
      };
      auto run = [&](auto m) {
        return mma_tile<decltype(m)::value>(nk, tmem, smem, ring, full, empty, tfull, tempty, uses,
                                            issued, abort_flag, err, fetch);
      };
      ok = mode == kFew    ? run(std::integral_constant<int, kFew>())
           : mode == kMore ? run(std::integral_constant<int, kMore>())
                           : run(std::integral_constant<int, kAll>());
    }
    if (issued) {  // make sure every MMA has retired before TMEM is released
      if (elect_one()) umma_commit(drain);
      __syncwarp();
      volatile int no_abort = 0;
      mbar_wait(drain, 0, &no_abort, err, 4);
    }
  } else {
    // ---------------- epilogue ----------------
    const Epilogue e{tfull, tempty, esync, abort_flag, last_part, axes, blocks, RA, RB,
                     A,     B,      C,     slots,      arrivals,  err,  tmem_base};
    uint32_t uses = 0;
    for (int64_t i = 0;; ++i) {
      const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
      if (pos >= ntiles) break;
      const Tile tr = tiles[pos];
      const Problem& P = probs[tr.prob];
      int nk = 0;
      int mode = kFew;
      if (pos < ntiles_k) {
        uint32_t w = info[i % kInfo];
        for (const long long t0 = clock64(); w >> 16 != (uint32_t)(i & 0xffff);
             w = info[i % kInfo]) {
          if (*abort_flag) break;
          if (clock64() - t0 > kWaitCycles) {
            *abort_flag = 1;
            record_wait(err, 7);
          }
        }
        if (!__all_sync(0xffffffffu, w >> 16 == (uint32_t)(i & 0xffff))) break;
        w = warp_uniform(w);
        nk = (int)(w & 0x1fffu);
        mode = (int)(w >> 13 & 3);
      }
      bool ok = true;
      if (mode == kAll) {
        const uint2 r = finish_tile_all<MAP>(e, tiles + pos, &P, nk, uses, parts);
        ok = r.x != 0;
        uses = r.y;
      } else {
        ok = finish_tile<MAP, false>(e, tr, P, nk, mode, uses, parts);
      }
      if (!ok) break;
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
// (with 1.5 for kCutSteps chi = 2048 took 2% longer, chi = 517 the same)
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
         round256(sizeof(int32_t) * (size_t)lA) + round256(sizeof(int32_t) * (size_t)lB) +
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
  int64_t tA = 0, tB = 0, rA = 0, rB = 0, lA = 0, lB = 0;
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
    P.lA = (int32_t)lA;
    P.lB = (int32_t)lB;
    lA += ceil_div(P.M, kRowBlock);
    lB += ceil_div(P.N, kRowBlock);
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
      for (int mi = 0; mi < P.mt; ++mi) {
        Tile x{p, mi, ni, 0, P.nk, 0, 1, (int32_t)P.K};
        x.rowA = (int32_t)((P.tA + (int64_t)mi * P.nk) * BM);
        x.rowB = (int32_t)((P.tB + (int64_t)ni * P.nk) * BN);
        x.lA = P.lA + mi * (BM / kRowBlock);
        x.lB = P.lB + ni * (BN / kRowBlock);
        x.nA = (int32_t)std::min<int64_t>(BM / kRowBlock, ceil_div(P.M - (int64_t)mi * BM, kRowBlock));
        x.nB = (int32_t)std::min<int64_t>(BN / kRowBlock, ceil_div(P.N - (int64_t)ni * BN, kRowBlock));
        t.tiles.push_back(x);
      }
    if (P.K > 0) {
      for (int64_t r = 0; r < P.M; r += kRowBlock) t.items.push_back(make_int2(p, (int)r));
      for (int64_t r = 0; r < P.N; r += kRowBlock)
        t.items.push_back(make_int2(p | (1 << 30), (int)r));
    }
    G.flops += 2.0 * x.M * x.N * x.K;
    if (!task.map) G.tasks.push_back(x);
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
      // (a long K at least as far as its sums fit 64 bits)
      const int parts = std::max<int>(std::min<int>(kMaxParts, (int)ceil_div(std::max(x.ks1, 1), most)),
                                      (int)ceil_div(x.ks1, kWideSteps));
      for (int q = 0; q < parts; ++q) {
        Tile y = x;
        y.ks0 = (int)((int64_t)x.ks1 * q / parts);
        y.ks1 = (int)((int64_t)x.ks1 * (q + 1) / parts);
        y.slot = (int32_t)slots;
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
  G.ntiles_k = std::count_if(t.tiles.begin(), t.tiles.end(), [](const Tile& x) { return x.ks1 > x.ks0; });
  G.nitems = (int)t.items.size();
  for (const Problem& P : t.probs) G.max_nk = std::max(G.max_nk, P.nk);
  G.rowsA = std::max<int64_t>(tA, 1) * BM;
  G.rowsB = std::max<int64_t>(tB, 1) * BN;
  G.rA = rA;
  G.rB = rB;
  G.lA = lA;
  G.lB = lB;
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
    table_bytes += img.bytes.size();
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
  table_bytes = 0;
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
  int32_t* LA = (int32_t*)((unsigned char*)RB + round256(sizeof(int32_t) * (size_t)G.rB));
  int32_t* LB = (int32_t*)((unsigned char*)LA + round256(sizeof(int32_t) * (size_t)G.lA));
  int* arrivals = (int*)((unsigned char*)LB + round256(sizeof(int32_t) * (size_t)G.lB));
  unsigned long long* slots =
      (unsigned long long*)((unsigned char*)arrivals + round256(sizeof(int) * (size_t)G.nslots));
  CUtensorMap tmA, tmB;
  make_slice_map(&tmA, packA, G.rowsA, kSlices, BM, BK, BK);
  make_slice_map(&tmB, packB, G.rowsB, kSlices, BN, BK, BK);
  set_smem_limit_once(ctx, smem_set, gemm_f64tc_kernel<MAP>, kSmemBytes);
  if (G.nitems) {
    KernelTimer timer(ctx, kKindPack);
    // CTAs per item: as many as keep an item's part in shared memory, and more while that fills the chip
    // (four CTAs fit an SM; a CTA's barriers and latencies are most of its time, two K steps each are
    // worth one). Left environment, chi = 1024, one-shot application, chi = 701, with eight CTAs per SM as
    // the limit / six / four: 150 / 145 / 143 us, 135 / 131 / 128.
    int ncta = 1;
    while (ncta < kMaxCluster &&
           (ceil_div(G.max_nk, ncta) > kCacheSteps ||
            (ceil_div(G.max_nk, ncta) > 2 && G.nitems * ncta * 2 <= 4 * ctx->num_sms)))
      ncta *= 2;
    const int steps = (int)std::min<int64_t>(kCacheSteps, ceil_div(G.max_nk, ncta));
    const int smem = steps * BK * kPadRows * (int)sizeof(double);
    set_smem_limit_once(ctx, pack_set, pack_f64_kernel<MAP>,
                        kCacheSteps * BK * kPadRows * (int)sizeof(double));
    launch_chained(pack_f64_kernel<MAP>, dim3((unsigned)G.nitems * (unsigned)ncta), dim3(256),
                   (size_t)smem, st, ncta, G.d_probs, G.d_items, ncta, steps, G.d_axes, G.d_blocks,
                   A, B, RA, RB, LA, LB, packA, packB, G.rowsA, G.rowsB, arrivals, (ulonglong2*)slots,
                   (int)G.nslots, parts.a,
                   parts.b);
    ctx->kernel_launches++;
  }
  KernelTimer timer(ctx, kKindGemmF64, G.flops);
  const int grid = (int)std::min<int64_t>(G.ntiles, ctx->num_sms);
  launch_chained(gemm_f64tc_kernel<MAP>, dim3((unsigned)grid), dim3(kThreads), (size_t)kSmemBytes, st,
                 1, tmA, tmB, G.d_probs, G.d_tiles, G.ntiles, G.ntiles_k, RA, RB, LA, LB, G.d_axes, G.d_blocks, A, B, C,
                 slots, arrivals, ctx->wait_err + kWaitGemm, parts);
  ctx->kernel_launches++;
}

bool launch(Context* ctx, Plan& p, const double* A, const double* B, double* C,
            const PartOffsets& parts) {
  cudaStream_t st = ctx->stream;
  for (Group& G : p.groups) {
    if (G.ntiles == 0) continue;
    unsigned char* mem = nullptr;
    const size_t need = G.scratch_bytes();
    const cudaError_t e = need > ctx->scratch_limit ? cudaErrorMemoryAllocation
                                                    : cudaMallocAsync((void**)&mem, need, st);
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
