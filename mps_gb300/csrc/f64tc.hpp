// FP64 grouped block GEMM on the tensor cores: host plan and launcher (kernels_f64tc.cu).
#pragma once

#include <cstddef>
#include <memory>
#include <vector>

#include "runtime.hpp"

namespace mpsg {
namespace f64tc {

constexpr int BM = 128, BN = 64, BK = 32;  // output tile and K step
constexpr int kSlices = 8;                 // 8-bit digits of a 62-bit fixed-point operand
constexpr int kChunkSteps = 8;             // K steps between drains (256 columns: see the kernel)
constexpr int64_t kMaxK = 65536;           // whole K summed in 64 bits (fits up to 2^18)

// One sector GEMM as the kernels see it: rows of the 128-row operand, rows of the 64-row operand
// and the output by element strides. Either operand of the contraction may be the 128-row one
// (swap: it is B, and the output is written transposed), whichever pads fewer tiles.
struct Problem {
  int64_t M, N, K;            // rows of the 128-row operand, of the 64-row operand, contracted
  int64_t oa, ars, aks;       // element (m, k) of the 128-row operand at oa + m ars + k aks
  int64_t ob, brs, bks;       // element (n, k) of the 64-row operand
  int64_t oc, crs, ccs;       // output (m, n)
  int64_t tA, tB, rA, rB;     // first packed tile and first exponent entry of each operand
  int32_t mt, nt, nk, swap;   // M tiles, N tiles, K steps
};

// Problems that are packed and multiplied by one pair of launches (their packed operands share
// one scratch allocation of at most about kGroupBytes, more only for a single larger problem).
struct Group {
  int nprob = 0, nitems = 0;
  int64_t ntiles = 0, rowsA = 0, rowsB = 0, rA = 0, rB = 0;
  double flops = 0;
  unsigned char* d_tables = nullptr;  // problems, output tiles, packing items
  Problem* d_probs = nullptr;
  int4* d_tiles = nullptr;
  int2* d_items = nullptr;
  std::vector<GemmTask> tasks;
  std::unique_ptr<DevGemmPlan> plain;  // FP64-pipe tables, built if the scratch cannot be had
  size_t scratch_bytes() const;
};

struct Plan {
  std::vector<Group> groups;
  cudaStream_t stream = nullptr;
  void build(const std::vector<GemmTask>& g, cudaStream_t st);
  void release();
  double flops() const;
  ~Plan() { release(); }
};

// Host half of build for one group: tables in launch order (checked on the CPU by tests).
struct GroupTables {
  std::vector<Problem> probs;
  std::vector<int4> tiles;  // (problem, M tile, N tile, K steps), decreasing K steps
  std::vector<int2> items;  // (problem | side << 30, first row)
};
void plan_group(const std::vector<GemmTask>& g, Group& G, GroupTables& t);

// Whether a sector GEMM runs on the tensor cores (see the rule in kernels_f64tc.cu).
bool eligible(const GemmTask& t);

void launch(Context* ctx, Plan& p, const double* A, const double* B, double* C);

}  // namespace f64tc
}  // namespace mpsg
