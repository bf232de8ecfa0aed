// Index maps of a contraction: where each element of the fused matrices of its sector GEMMs lives
// in the operand and result tensors, so that kernels read blocks in place and write the result in
// place (no fused copies). Pure host code.
//
// A fused axis (rows, columns or contracted index of one sector GEMM) is a run of "combos": one per
// choice of leg charges, each a column-major run over its legs' states. A block of a tensor is the
// rectangle of one row combo and one column combo; within it an element's address is affine in
// the leg indices.
#pragma once

#include "planner.hpp"

namespace mpsg {

constexpr int kMapLegs = 3;  // legs per fused axis that a map can describe

// One index of a fused axis (16 bytes, read as an int4): its combo, the indices of its legs, and how
// many entries from this one on (itself included, at most 255) belong to the same combo with leg 0
// counting up, so that their addresses have one stride.
struct AxisEntry {
  int32_t combo_run;  // combo | run << 24
  int32_t i[kMapLegs];
};
constexpr int32_t kComboMask = 0xffffff;

// A block: address of its first element and the strides of the row-axis and column-axis legs.
// Offsets within a block stay below 2^31: kernels form them in 32 bits, 64-bit multiplications being
// several times slower on this chip.
struct MapBlock {
  int64_t base;
  int32_t rs[kMapLegs], cs[kMapLegs];
};

// One combo of a fused axis: first index, number of indices, leg sizes. Leg 0, which counts fastest,
// is the axis' longest leg, whatever the order of the legs in the tensors: a sector GEMM may take
// its rows, columns and contracted index in any order.
struct AxisCombo {
  int32_t start, count;
  int32_t d[kMapLegs];
};

// One sector GEMM. Block tables: A [row combo][k combo], B [column combo][k combo] (its column legs
// as rs, contracted legs as cs), C [row combo][column combo]. K = 0: the result block is zero.
struct MapProblem {
  int64_t M = 0, N = 0, K = 0;
  std::vector<AxisCombo> m, n, k;
  std::vector<MapBlock> A, B, C;
};

// Empty when the contraction cannot be mapped (more than kMapLegs legs on an axis, a block of 2^31
// elements, a scalar result).
std::vector<MapProblem> build_contract_map(const ContractPlan& p, const TensorMeta& A,
                                           const TensorMeta& B);

// Bits of a block's base that name the tensor it is in, where an operand or the result is several
// tensors of one structure (real and imaginary parts): part 0 has the pointer of a launch, the
// others are at distances (in elements) given with it.
constexpr int kPartShift = 61;
struct PartOffsets {
  int64_t a = 0, b = 0;          // from the real to the imaginary part of A, of B
  int64_t c1 = 0, c2 = 0, c3 = 0;  // from part 0 of the result to the others
};

// The map of the products of all parts of A and B, in the parts of A that have an imaginary one (ca)
// stacked along the rows and those of B (cb) along the columns. Part of the result: 2 [imaginary part of
// A] + [imaginary part of B] for two complex operands, else the part of the complex one.
// Empty when an axis gets too long.
std::vector<MapProblem> complex_map(const std::vector<MapProblem>& map, bool ca, bool cb);

#ifdef __CUDACC__
__device__ __forceinline__ int64_t part_base(int64_t base, int64_t d1, int64_t d2, int64_t d3) {
  const int part = (int)(base >> kPartShift);
  if (part) base = (base & (((int64_t)1 << kPartShift) - 1)) + (part == 1 ? d1 : part == 2 ? d2 : d3);
  return base;
}
#endif

// Appends the entries of an axis.
void append_axis(const std::vector<AxisCombo>& combos, std::vector<AxisEntry>& out);

}  // namespace mpsg
