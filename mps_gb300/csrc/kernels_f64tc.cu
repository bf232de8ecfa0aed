// FP64 grouped block GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), FP64 in,
// FP64-accurate out.
//
// GB300 issues 2 FP64 FMAs per SM and clock (1.1 TFLOP/s measured with cuBLAS), so a sector GEMM
// on the FP64 pipe is bound by it from a few blocks on. Here every operand row is written as
// 62-bit fixed point relative to its largest element and cut into eight balanced 8-bit digits,
// each exact in bf16; the digit products run on the tensor cores and are summed exactly:
//
//   * Packing (pack_f64_kernel). For row r of an operand (row of A, column of B) with |x| < 2^e,
//     F = round(x 2^(62-e)) = sum_p t_p 2^(8 (7-p)), |t_0| <= 64, -128 <= t_p <= 127; slice p
//     stores t_p 2^(-8p) as bf16. The digits come from the bytes of F + 0x0080808080808080.
//   * MMA. Slice pair (p, q) with p + q <= 7 belongs to group g = p + q, of weight 2^(-8g); 36
//     pairs. Groups 0..5 have a TMEM accumulator each, groups 6 and 7 share one: 7 x 64 = 448 of
//     the 512 columns. One K index adds at most 2^16 units of 2^(-8g) to a group g <= 4, so over
//     a chunk of 256 its FP32 sum is an exact integer below 2^24. Group 5 could reach 5/4 of
//     that (only if every digit had its largest value), and the shared accumulator rounds at
//     2^-24 of a sum of weight 2^-48: both far below the last bit of the result.
//   * Drain. After each chunk the epilogue warps add groups 0..4 as integers into one 64-bit
//     fixed-point sum per output element (unit 2^-32; K 2^12.03 products fit for K up to 2^18)
//     and the smaller groups into one FP32 sum, whose rounding is 2^-24 of a sum of weight 2^-40.
//     After the last chunk both are rounded to FP64 once. No FP64 instruction is issued.
//
// Every operand element is off by at most 2^-63 of its row's largest, products of weight 2^-64 and
// less are left out, and the result is rounded once, where a chain of K FP64 FMAs rounds K times.
//
// A row with a non-finite element, or whose largest element is outside 2^-400..2^400, is marked
// in its exponent; every output element of such a row or column is computed in the epilogue by
// the chain of FP64 FMAs over k, as the FP64-pipe kernel does, so NaN, infinities, overflow and
// subnormals come out as there.
//
// Tile 128 x 64: seven accumulators of 64 columns fill TMEM. The MMAs are bound by shared-memory
// operand reads (6 KB per 32-cycle MMA).
//
// Measured (two-site H_eff, GEMMs of one application, FP64 pipe -> packing + this kernel):
// chi = 2048, 8.9 GFLOP: 9205 -> 99 + 437 us; chi = 517: 870 -> 30 + 80 us; chi = 48 (K about
// 20): 110 -> 11 + 31 us. Relative error of N(0,1) products against extended precision: 2e-16
// (K = 33) to 1.4e-15 (K = 2050) on the FP64 pipe, 5e-17 here.
#include <cuda_bf16.h>

#include <algorithm>

#include "f64tc.hpp"
#include "tc5.cuh"

namespace mpsg {
namespace f64tc {

using namespace tc;

namespace {

constexpr int kAccs = 7;
constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2;
constexpr int kStageBytes = kSlices * (kABytes + kBBytes);  // 96 KB
constexpr int kStages = 2;
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
constexpr int kTmemCols = 512;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kEpiCols = BN * 4 / kEpiWarps;  // 16 columns per epilogue thread

constexpr int kRowZero = 1 << 20;  // exponent entry of an all-zero row
constexpr int kRowBad = 1 << 21;   // ... of a row outside the sliced range (see above)
constexpr int kExpRange = 400;
constexpr int kRowBlock = 32;      // rows per packing item

// Adds one accumulator element of an exact group G <= 4 (v a multiple of 2^(-8G)) into a 64-bit sum
// in units of 2^-32.
template <int G>
__device__ __forceinline__ void add_group(long long& hi, float v) {
  const int i = __float2int_rn(v * (float)(1u << (8 * G < 32 ? 8 * G : 0)) *
                               (8 * G < 32 ? 1.f : 4294967296.f));
  if constexpr (G == 0) hi += (long long)((unsigned long long)(unsigned)i << 32);
  else hi += (long long)i * (long long)(1 << (32 - 8 * G));
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

// Adds one chunk's seven accumulators into 8 elements of (hi, lo); taddr = first column of the
// group-0 accumulator in this warp's TMEM lanes.
__device__ __forceinline__ void drain8(uint32_t taddr, long long* hi, float* lo) {
  uint32_t v[2][8];
#pragma unroll
  for (int g = 0; g < kAccs; g += 2) {  // two accumulators at a time: few registers live
    tmem_ld8(taddr + g * BN, v[0]);
    if (g + 1 < kAccs) tmem_ld8(taddr + (g + 1) * BN, v[1]);
    tmem_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = __uint_as_float(v[0][j]), y = __uint_as_float(v[1][j]);
      if (g == 0) {
        add_group<0>(hi[j], x);
        add_group<1>(hi[j], y);
      } else if (g == 2) {
        add_group<2>(hi[j], x);
        add_group<3>(hi[j], y);
      } else if (g == 4) {
        add_group<4>(hi[j], x);
        lo[j] += y;
      } else {
        lo[j] += x;
      }
    }
  }
}

// (hi 2^-32 + lo) 2^E rounded to nearest even (integer instructions; the result is in the normal
// range). hi moves up by the free bits it has, at most 24, before lo joins it.
__device__ __forceinline__ double sum_to_f64(long long hi, float lo, int E) {
  const unsigned long long mag = hi < 0 ? 0ull - (unsigned long long)hi : (unsigned long long)hi;
  const int sh = max(0, min(24, __clzll((long long)mag) - 2));
  const long long a = (long long)((unsigned long long)hi << sh) +
                      __float2ll_rn(lo * __uint_as_float((uint32_t)(127 + 32 + sh) << 23));
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
  bits += (unsigned long long)(63 - lz - 32 - sh + E + 1023) << 52;
  return __longlong_as_double((long long)(sign | bits));
}

// One CTA per item: 32 rows of one operand, whole K: the rows' exponents first, then their
// digits. Work per element is about 35 integer and FP32 instructions against 8 bytes read and 16
// written; the second read of an item mostly hits the L1 or L2.
__global__ void __launch_bounds__(256) pack_f64_kernel(
    const Problem* __restrict__ probs, const int2* __restrict__ items, int nitems,
    const double* __restrict__ A, const double* __restrict__ B, int32_t* __restrict__ RA,
    int32_t* __restrict__ RB, __nv_bfloat16* __restrict__ packA, __nv_bfloat16* __restrict__ packB,
    int64_t rowsA, int64_t rowsB) {
  __shared__ unsigned long long red[8][33];
  __shared__ int rexp[kRowBlock];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int2 item = items[it];
    const int side = (item.x >> 30) & 1;
    const Problem P = probs[item.x & 0x3fffffff];
    const int64_t r0 = item.y;
    const int64_t rows = side ? P.N : P.M, rs = side ? P.brs : P.ars, ks = side ? P.bks : P.aks;
    const double* X = (((P.swap != 0) != (side != 0)) ? B : A) + (side ? P.ob : P.oa);
    const int nr = (int)min((int64_t)kRowBlock, rows - r0);
    // exponents: lanes along whichever axis is contiguous
    if (rs == 1) {
      unsigned long long m = 0;
      if (lane < nr)
        for (int64_t k = w; k < P.K; k += 8) {
          const unsigned long long b =
              (unsigned long long)__double_as_longlong(X[r0 + lane + k * ks]) & ~(1ull << 63);
          m = b > m ? b : m;
        }
      red[w][lane] = m;
    } else {
      for (int rr = w; rr < kRowBlock; rr += 8) {
        unsigned long long m = 0;
        if (rr < nr)
          for (int64_t k = lane; k < P.K; k += 32) {
            const unsigned long long b =
                (unsigned long long)__double_as_longlong(X[(r0 + rr) * rs + k * ks]) &
                ~(1ull << 63);
            m = b > m ? b : m;
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long q = __shfl_xor_sync(0xffffffffu, m, o);
          m = q > m ? q : m;
        }
        if (lane < 8) red[lane][rr] = lane == 0 ? m : 0;
      }
    }
    __syncthreads();
    if (t < kRowBlock) {
      unsigned long long m = 0;
#pragma unroll
      for (int g = 0; g < 8; ++g) m = red[g][t] > m ? red[g][t] : m;
      int e = (int)(m >> 52) - 1022;  // |x| < 2^e for the row's largest |x|
      if (m == 0) e = kRowZero;
      else if (e < -kExpRange || e > kExpRange) e = kRowBad;  // also Inf and NaN
      rexp[t] = e;
      if (t < nr) (side ? RB + P.rB : RA + P.rA)[r0 + t] = e;
    }
    __syncthreads();
    // digits: a warp covers 8 rows x 32 K of one step, a thread 8 consecutive K of a row
    const int rr = (w & 3) * 8 + (lane >> 2), g8 = (lane & 3) * 8;
    const int rpt = side ? BN : BM;
    const int64_t r = r0 + rr;
    const int64_t tile0 = (side ? P.tB : P.tA) + (r / rpt) * P.nk;
    const int64_t plane = (side ? rowsB : rowsA) * BK;
    __nv_bfloat16* out = side ? packB : packA;
    const int e = rexp[rr];
    if (rr < nr) {
      for (int s = w >> 2; s < P.nk; s += 2) {
        const int64_t k0 = (int64_t)s * BK + g8;
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = k0 + j < P.K ? __ldg(X + r * rs + (k0 + j) * ks) : 0.0;
        uint32_t packed[kSlices][4];
        float prev[kSlices];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int hw = __double2hiint(x[j]);
          const uint32_t lw = (uint32_t)__double2loint(x[j]);
          const int eb = (hw >> 20) & 0x7ff;
          const int d = e + 1022 - eb;  // >= 0 in a row of the sliced range
          const unsigned long long m =
              ((((unsigned long long)((uint32_t)hw & 0xfffffu)) << 32 | lw) | (1ull << 52)) << 9;
          long long F = 0;
          if (eb != 0 && d >= 0 && d <= 62) {
            F = (long long)((m + ((1ull << d) >> 1)) >> d);
            if (hw < 0) F = -F;
          }
          const unsigned long long G = (unsigned long long)F + 0x8080808080808080ull;
          const uint32_t gh = (uint32_t)(G >> 32), gl = (uint32_t)G;
#pragma unroll
          for (int q = 0; q < kSlices; ++q) {
            // byte b of digit q (offset by 128) as the low mantissa bits of 2^(23 - 8q)
            const uint32_t magic = (uint32_t)(150 - 8 * q) << 23;
            const uint32_t f = __byte_perm(q < 4 ? gh : gl, magic, 0x7650 | (3 - (q & 3)));
            const float v = __uint_as_float(f) - __uint_as_float(magic | 128u);
            if (j & 1) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(prev[q], v);  // exact
              packed[q][j >> 1] = *reinterpret_cast<const uint32_t*>(&h);
            } else {
              prev[q] = v;
            }
          }
        }
        const int64_t idx = ((tile0 + s) * rpt + (r % rpt)) * BK + g8;
#pragma unroll
        for (int q = 0; q < kSlices; ++q)
          *reinterpret_cast<uint4*>(out + q * plane + idx) =
              make_uint4(packed[q][0], packed[q][1], packed[q][2], packed[q][3]);
      }
    }
    __syncthreads();  // rexp and red are rewritten by the next item
  }
}

// Persistent, one CTA per SM: warp 0 TMA producer, warp 1 TMEM allocator and MMA issuer, 16
// epilogue warps (four per TMEM lane quarter, 16 columns each). Every mbarrier wait is bounded;
// on expiry the kernel records an error code, stops issuing, waits for its own MMAs and frees
// TMEM.
__global__ void __launch_bounds__(kThreads, 1) gemm_f64tc_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
    const Problem* __restrict__ probs, const int4* __restrict__ tiles, int64_t ntiles,
    const int32_t* __restrict__ RA, const int32_t* __restrict__ RB, const double* __restrict__ A,
    const double* __restrict__ B, double* __restrict__ C, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + kStages * kStageBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kStages;
  uint64_t* tfull = bars + 2 * kStages;
  uint64_t* tempty = tfull + 1;
  uint64_t* drain = tempty + 1;
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 32 * kEpiWarps);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int64_t i = 0; !*abort_flag; ++i) {
        const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
        if (pos >= ntiles) break;
        const int4 tr = tiles[pos];
        const int nk = tr.w;
        const int rowA = (int)((probs[tr.x].tA + (int64_t)tr.y * nk) * BM);
        const int rowB = (int)((probs[tr.x].tB + (int64_t)tr.z * nk) * BN);
        for (int ks = 0; ks < nk; ++ks) {
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
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(BM, BN);
      int stage = 0;
      uint32_t phase = 0, use = 0;
      bool issued = false;
      for (int64_t i = 0; !*abort_flag; ++i) {
        const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
        if (pos >= ntiles) break;
        const int nk = tiles[pos].w;
        for (int c0 = 0; c0 < nk && !*abort_flag; c0 += kChunkSteps) {
          if (!mbar_wait(tempty, (use & 1) ^ 1, abort_flag, err, 2)) break;
          tc_fence_after();
          uint32_t init = 0;  // bit g: accumulator g already written in this chunk
          const int c1 = min(nk, c0 + kChunkSteps);
          for (int ks = c0; ks < c1; ++ks) {
            if (!mbar_wait(&full[stage], phase, abort_flag, err, 3)) break;
            tc_fence_after();
            const uint32_t sA = smem_u32(smem + stage * kStageBytes);
            const uint32_t sB = sA + kSlices * kABytes;
#pragma unroll
            for (int pa = 0; pa < kSlices; ++pa) {
#pragma unroll
              for (int qb = 0; qb < kSlices - pa; ++qb) {
                const int g = pa + qb < kAccs ? pa + qb : kAccs - 1;
                const uint64_t ad = sw64_desc(sA + pa * kABytes);
                const uint64_t bd = sw64_desc(sB + qb * kBBytes);
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) {
                  umma_bf16(tmem_base + (uint32_t)(g * BN), ad + 2 * kk, bd + 2 * kk, idesc,
                            (init >> g) & 1u);
                  init |= 1u << g;
                }
              }
            }
            umma_commit(&empty[stage]);
            issued = true;
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
          }
          umma_commit(tfull);
          ++use;
        }
      }
      if (issued) {  // make sure every MMA has retired before TMEM is released
        umma_commit(drain);
        volatile int no_abort = 0;
        mbar_wait(drain, 0, &no_abort, err, 4);
      }
    }
  } else {
    // ---------------- epilogue ----------------
    const int lrow = 32 * (warp & 3) + lane;  // TMEM lane = tile row
    const int col0 = ((warp - 2) >> 2) * kEpiCols;
    const uint32_t taddr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
    uint32_t use = 0;
    for (int64_t i = 0;; ++i) {
      const int64_t pos = sched_pos(i, gridDim.x, blockIdx.x);
      if (pos >= ntiles) break;
      const int4 tr = tiles[pos];
      const Problem& P = probs[tr.x];
      const int64_t K = P.K;
      long long hi[kEpiCols];
      float lo[kEpiCols];
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j) {
        hi[j] = 0;
        lo[j] = 0.f;
      }
      bool ok = true;
      for (int c0 = 0; c0 < tr.w; c0 += kChunkSteps) {
        if (!mbar_wait(tfull, use & 1, abort_flag, err, 5)) {
          ok = false;
          break;
        }
        tc_fence_after();
        drain8(taddr, hi, lo);
        drain8(taddr + 8, hi + 8, lo + 8);
        tc_fence_before();
        mbar_arrive(tempty);
        ++use;
      }
      if (!ok) break;
      const int64_t row = (int64_t)tr.y * BM + lrow;
      if (row < P.M) {
        const int64_t n0 = (int64_t)tr.z * BN + col0;
        const int nc = (int)min((int64_t)kEpiCols, P.N - n0);
        const int er = K ? RA[P.rA + row] : kRowZero;
        const int32_t* RBp = RB + P.rB + n0;
        double* Cp = C + P.oc + row * P.crs + n0 * P.ccs;
        const int64_t ccs = P.ccs;
#pragma unroll
        for (int j = 0; j < kEpiCols; ++j) {
          if (j >= nc) break;
          const int ec = K ? RBp[j] : kRowZero;
          double y;
          if (er >= kRowZero || ec >= kRowZero) {
            y = 0.0;
            if (er == kRowBad || ec == kRowBad) {  // the FMA chain (not sliced)
              const double* Xa = (P.swap ? B : A) + P.oa + row * P.ars;
              const double* Xb = (P.swap ? A : B) + P.ob + (n0 + j) * P.brs;
              for (int64_t k = 0; k < K; ++k) y = fma(Xa[k * P.aks], Xb[k * P.bks], y);
            }
          } else {
            y = sum_to_f64(hi[j], lo[j], er + ec - 12);
          }
          Cp[j * ccs] = y;
        }
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

size_t round256(size_t n) { return (n + 255) & ~size_t(255); }

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

size_t packed_bytes(const GemmTask& t) {
  return (size_t)(ceil_div(t.M, BM) * BM + ceil_div(t.N, BN) * BN + 128) *
         (size_t)(ceil_div(t.K, BK) * BK) * 2 * kSlices;
}

}  // namespace

// Every tiled task (K > 32, or M and N > 32) is faster here, down to the smallest: a 64 x 64 tile
// takes the FP64 pipe 2048 cycles per k index, whatever part of it is padding, and the tensor
// cores about 36 x 3 (chi = 48: 55 us a GEMM against 21 with its packing). Beyond kMaxK the
// 64-bit sums could overflow; such a K is left to the FP64 pipe.
bool eligible(const GemmTask& t) { return t.K <= kMaxK; }

size_t Group::scratch_bytes() const {
  return round256((size_t)rowsA * BK * 2 * kSlices) + round256((size_t)rowsB * BK * 2 * kSlices) +
         round256(sizeof(int32_t) * (size_t)rA) + round256(sizeof(int32_t) * (size_t)rB);
}

void plan_group(const std::vector<GemmTask>& g, Group& G, GroupTables& t) {
  int64_t tA = 0, tB = 0, rA = 0, rB = 0;
  G.flops = 0;
  for (const GemmTask& x : g) {
    Problem P;
    // the operand with more rows per padded tile takes the 128-row side: fewer output tiles, then
    // fewer packed rows
    const int64_t direct = ceil_div(x.M, BM) * ceil_div(x.N, BN);
    const int64_t swapped = ceil_div(x.N, BM) * ceil_div(x.M, BN);
    P.swap = swapped < direct ? 1 : 0;
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
    const int p = (int)t.probs.size();
    for (int ni = 0; ni < P.nt; ++ni)
      for (int mi = 0; mi < P.mt; ++mi) t.tiles.push_back(make_int4(p, mi, ni, P.nk));
    if (P.K > 0) {
      for (int64_t r = 0; r < P.M; r += kRowBlock) t.items.push_back(make_int2(p, (int)r));
      for (int64_t r = 0; r < P.N; r += kRowBlock)
        t.items.push_back(make_int2(p | (1 << 30), (int)r));
    }
    G.flops += 2.0 * x.M * x.N * x.K;
    t.probs.push_back(P);
  }
  std::stable_sort(t.tiles.begin(), t.tiles.end(),
                   [](const int4& a, const int4& b) { return a.w > b.w; });
  std::stable_sort(t.items.begin(), t.items.end(), [&](const int2& a, const int2& b) {
    return t.probs[a.x & 0x3fffffff].K > t.probs[b.x & 0x3fffffff].K;
  });
  G.tasks = g;
  G.nprob = (int)t.probs.size();
  G.ntiles = (int64_t)t.tiles.size();
  G.nitems = (int)t.items.size();
  G.rowsA = std::max<int64_t>(tA, 1) * BM;
  G.rowsB = std::max<int64_t>(tB, 1) * BN;
  G.rA = rA;
  G.rB = rB;
}

void Plan::build(const std::vector<GemmTask>& g, cudaStream_t st) {
  release();
  stream = st;
  std::vector<std::vector<GemmTask>> parts;
  size_t bytes = 0;
  for (const GemmTask& t : g) {
    const size_t b = packed_bytes(t);
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
    plan_group(part, G, t);
    const size_t bp = round256(sizeof(Problem) * t.probs.size()),
                 bt = round256(sizeof(int4) * t.tiles.size()),
                 bi = round256(sizeof(int2) * t.items.size());
    std::vector<unsigned char> img(bp + bt + bi);
    std::copy_n((const unsigned char*)t.probs.data(), sizeof(Problem) * t.probs.size(), img.data());
    std::copy_n((const unsigned char*)t.tiles.data(), sizeof(int4) * t.tiles.size(),
                img.data() + bp);
    if (!t.items.empty())
      std::copy_n((const unsigned char*)t.items.data(), sizeof(int2) * t.items.size(),
                  img.data() + bp + bt);
    MPSG_CUDA(cudaMallocAsync((void**)&G.d_tables, img.size(), st));
    MPSG_CUDA(cudaMemcpyAsync(G.d_tables, img.data(), img.size(), cudaMemcpyHostToDevice, st));
    G.d_probs = (Problem*)G.d_tables;
    G.d_tiles = (int4*)(G.d_tables + bp);
    G.d_items = (int2*)(G.d_tables + bp + bt);
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

void launch(Context* ctx, Plan& p, const double* A, const double* B, double* C) {
  static std::once_flag smem_set[kMaxDevices];
  cudaStream_t st = ctx->stream;
  for (Group& G : p.groups) {
    if (G.ntiles == 0) continue;
    unsigned char* mem = nullptr;
    const cudaError_t e = cudaMallocAsync((void**)&mem, G.scratch_bytes(), st);
    if (e == cudaErrorMemoryAllocation) {
      // no room for the packed operands (twice the FP64 ones): the FP64-pipe kernel needs none
      (void)cudaGetLastError();
      if (!G.plain) {
        G.plain = std::make_unique<DevGemmPlan>();
        G.plain->upload(G.tasks, G.flops, st, false);
      }
      launch_gemm_f64(ctx, *G.plain, A, B, C);
      ctx->gemm_flops -= G.flops;  // counted by the caller
      continue;
    }
    MPSG_CUDA(e);
    const size_t bA = round256((size_t)G.rowsA * BK * 2 * kSlices),
                 bB = round256((size_t)G.rowsB * BK * 2 * kSlices);
    __nv_bfloat16* packA = (__nv_bfloat16*)mem;
    __nv_bfloat16* packB = (__nv_bfloat16*)(mem + bA);
    int32_t* RA = (int32_t*)(mem + bA + bB);
    int32_t* RB = (int32_t*)(mem + bA + bB + round256(sizeof(int32_t) * (size_t)G.rA));
    CUtensorMap tmA, tmB;
    make_slice_map(&tmA, packA, G.rowsA, kSlices, BM, BK, BK);
    make_slice_map(&tmB, packB, G.rowsB, kSlices, BN, BK, BK);
    set_smem_limit_once(ctx, smem_set, gemm_f64tc_kernel, kSmemBytes);
    if (G.nitems) {
      KernelTimer timer(ctx, kKindPack);
      const int grid = std::min(G.nitems, ctx->num_sms * 8);
      pack_f64_kernel<<<grid, 256, 0, st>>>(G.d_probs, G.d_items, G.nitems, A, B, RA, RB, packA,
                                           packB, G.rowsA, G.rowsB);
      MPSG_CUDA(cudaGetLastError());
      ctx->kernel_launches++;
    }
    {
      KernelTimer timer(ctx, kKindGemmF64, G.flops);
      const int grid = (int)std::min<int64_t>(G.ntiles, ctx->num_sms);
      gemm_f64tc_kernel<<<grid, kThreads, kSmemBytes, st>>>(tmA, tmB, G.d_probs, G.d_tiles,
                                                            G.ntiles, RA, RB, A, B, C,
                                                            ctx->d_tc_err);
      MPSG_CUDA(cudaGetLastError());
      ctx->kernel_launches++;
    }
    MPSG_CUDA(cudaFreeAsync(mem, st));
  }
  if (ctx->debug_sync) {
    int code = 0;
    MPSG_CUDA(cudaMemcpyAsync(&code, ctx->d_tc_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    MPSG_CUDA(cudaStreamSynchronize(st));
    if (code) {
      MPSG_CUDA(cudaMemsetAsync(ctx->d_tc_err, 0, sizeof(int), st));
      throw Error(kErrCuda, "FP64 tensor-core GEMM: a bounded wait expired (role code " +
                                std::to_string(code) + ")");
    }
  }
}

}  // namespace f64tc
}  // namespace mpsg
