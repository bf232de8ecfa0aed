// FP64 contraction without fused copies: sector GEMMs that read the operand tensors and write the
// result tensor in place through index maps (kernels_map.cu, kernels_f64tc.cu).
#pragma once

#include "contract_map.hpp"
#include "f64tc.hpp"

namespace mpsg {

// One sector GEMM of the element-per-thread kernel (block tables as in MapProblem).
struct SmallProblem {
  int32_t first, mt;         // first tile (rows fastest) of the launch, tiles along the rows
  int32_t M, N, K;
  int32_t axM, axN, axK;     // first axis entries
  int32_t nkc, nnc;          // k combos, column combos
  int32_t blkA, blkB, blkC;  // first blocks
};

// Offsets from a block's rows: element (i0, i1, i2) of the long axis at off + i0 rs0 + i1 rs1 + i2 rs2.
struct alignas(16) ThinOffset {
  int64_t off;
  int32_t rs0, rs1, rs2, pad;
};

// Rows [start, start + count) of one combo of the long axis of a thin sector GEMM: L is the operand
// with the long axis, T (the thin axis) and K are at most kThinMax.
struct alignas(16) ThinUnit {
  int32_t T, K, longB;      // longB: L is B (the long axis is the columns)
  int32_t offs;             // K offsets into L, then T offsets into the output
  int32_t vals;             // T x K positions of the thin operand's elements
  int32_t start, count;
  uint32_t d0, m0, s0, d1, m1, s1;  // sizes and division constants of the first two legs
  int32_t pad[3];
};

constexpr int kThinMax = 32;

struct DirectTables {
  std::vector<SmallProblem> small;
  std::vector<ThinUnit> units;
  std::vector<ThinOffset> offs;
  std::vector<int64_t> vals;
  std::vector<AxisEntry> axes;
  std::vector<MapBlock> blocks;
  int64_t small_tiles = 0;        // of the small problems
  std::vector<f64tc::Task> tiled; // points into the map it was planned from
};

struct DirectPlan {
  unsigned char* d_tables = nullptr;
  size_t table_bytes = 0;
  cudaStream_t stream = nullptr;
  SmallProblem* d_small = nullptr;
  ThinUnit* d_units = nullptr;
  ThinOffset* d_offs = nullptr;
  int64_t* d_vals = nullptr;
  AxisEntry* d_axes = nullptr;
  MapBlock* d_blocks = nullptr;
  int nsmall = 0, small_tiles = 0, nunits = 0, thin_k = 0;
  double flops = 0, tc_flops = 0;
  std::unique_ptr<f64tc::Plan> tc;
  // false: the contraction cannot be mapped, or the fused path is the better one for it
  // ca, cb: A, B have imaginary parts (the products of all parts in one set of launches)
  bool build(const ContractPlan& p, const TensorMeta& A, const TensorMeta& B, int num_sms,
             cudaStream_t st, bool ca, bool cb);
  size_t device_bytes() const { return table_bytes + (tc ? tc->table_bytes : 0); }
  ~DirectPlan();
};

// Host half of build: which kernel takes each sector GEMM, and its tables (checked on the CPU).
void plan_direct(const std::vector<MapProblem>& map, const std::vector<GemmTask>& gemms,
                 int num_sms, DirectTables& t);

// C = contract(A, B); false (nothing useful written) when scratch for the tensor cores could not be
// had.
bool launch_direct(Context* ctx, DirectPlan& p, const double* A, const double* B, double* C,
                   const PartOffsets& parts = PartOffsets());

// re = rr + c_ii ii in place of rr, im = c_ri ri + c_ir ir in place of ri
void launch_complex_parts(Context* ctx, int64_t n, double* rr, double* ri, const double* ir,
                          const double* ii, double c_ri, double c_ir, double c_ii);

}  // namespace mpsg
