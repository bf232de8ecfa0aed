// FP64 grouped block GEMM on the tensor cores: host plan and launcher (kernels_f64tc.cu).
#pragma once

#include <cstddef>
#include <memory>
#include <vector>

#include "contract_map.hpp"
#include "runtime.hpp"

namespace mpsg {
namespace f64tc {

constexpr int BM = 128, BN = 64, BK = 32;  // output tile and K step
constexpr int kSlices = 9;                 // 9-bit digits of a 79-bit fixed-point operand
constexpr int kFewSlices = 7;              // the leading ones, which most tiles need
constexpr int64_t kMaxK = 65536;           // whole K summed in 64 bits (fits up to 2^22)

// One sector GEMM as the kernels see it: R is the operand on the 128-row side, S the one on the
// 64-row side. Either operand of the contraction may be R (swap: it is B, and the output is written
// transposed), see plan_group. Elements are found by strides (fused matrices) or, in a
// mapped group, by axis entries and block tables (the tensors themselves).
struct Problem {
  int64_t M, N, K;            // rows of R, rows of S, contracted
  int64_t oa, ars, aks;       // element (m, k) of R at oa + m ars + k aks
  int64_t ob, brs, bks;       // element (n, k) of S
  int64_t oc, crs, ccs;       // output (m, n)
  int64_t tA, tB, rA, rB;     // first packed tile and first exponent entry of each operand
  int32_t lA, lB;             // first count of large elements (one per 32 rows), R and S
  int32_t mt, nt, nk, swap;   // M tiles, N tiles, K steps
  int32_t axM, axN, axK;      // mapped: first axis entry of the rows of R, of S and of k
  int32_t blkA, blkB, blkC;   // ... first block of R [row combo][k combo], of S, of the output
  int32_t nkc, nnc;           // ... k combos, combos of the rows of S
  int32_t fastA, fastB;       // rows (1) or k (0) contiguous in memory
};

// One output tile, or one of `parts` pieces of its K steps: the pieces add their sums to scratch slot
// `slot` and the last one to arrive writes the tile.
struct alignas(16) Tile {
  int32_t prob, mi, ni, ks0, ks1;  // K steps [ks0, ks1)
  int32_t slot, parts;
  int32_t K;                       // of the problem
  int32_t lA, lB, nA, nB;          // counts of large elements of its rows: first and number, R and S
  int32_t rowA, rowB;              // first packed row of K step 0, R and S
};

// Problems that are packed and multiplied by one pair of launches (their packed operands share
// one scratch allocation of at most about kGroupBytes, more only for a single larger problem).
struct Group {
  int nprob = 0, nitems = 0, max_nk = 0;
  int64_t ntiles = 0, ntiles_k = 0;  // ntiles_k: those with K steps, which come first
  int64_t nslots = 0, rowsA = 0, rowsB = 0, rA = 0, rB = 0, lA = 0, lB = 0;
  double flops = 0;
  unsigned char* d_tables = nullptr;  // problems, output tiles, packing items
  Problem* d_probs = nullptr;
  Tile* d_tiles = nullptr;
  int2* d_items = nullptr;
  AxisEntry* d_axes = nullptr;   // mapped groups only
  MapBlock* d_blocks = nullptr;
  std::vector<GemmTask> tasks;         // not of a mapped plan, whose caller has another way
  std::unique_ptr<DevGemmPlan> plain;  // FP64-pipe tables of them, built if the scratch cannot be had
  size_t scratch_bytes() const;
};

// One sector GEMM of a plan: strides (GemmTask), and the index map when it reads tensors in place.
struct Task {
  GemmTask g;
  const MapProblem* map = nullptr;
};

struct Plan {
  std::vector<Group> groups;
  cudaStream_t stream = nullptr;
  bool mapped = false;
  size_t table_bytes = 0;  // on the device
  void build(const std::vector<Task>& g, int num_sms, cudaStream_t st);
  void release();
  double flops() const;
  ~Plan() { release(); }
};

// Host half of build for one group: tables in launch order (checked on the CPU by tests).
struct GroupTables {
  std::vector<Problem> probs;
  std::vector<Tile> tiles;  // decreasing K steps
  std::vector<int2> items;  // (problem | side << 30, first row)
  std::vector<AxisEntry> axes;
  std::vector<MapBlock> blocks;
};
void plan_group(const std::vector<Task>& g, int num_sms, Group& G, GroupTables& t);

// Whether a sector GEMM runs on the tensor cores (see the rule in kernels_f64tc.cu).
bool eligible(const GemmTask& t);

// C = A B for every problem of the plan. A plan whose operands are fused matrices falls back on the
// FP64 pipe where the packed operands find no memory; a mapped one returns false then, with
// nothing written that a rerun would not write again.
bool launch(Context* ctx, Plan& p, const double* A, const double* B, double* C,
            const PartOffsets& parts = PartOffsets());

}  // namespace f64tc
}  // namespace mpsg
