// Thin SVD of small blocks: column-pivoted Householder QR, A P = Q R, then one-sided Jacobi on R^T (plane
// rotations of column pairs until all columns are orthogonal: their norms are the singular values, the
// normalised columns the right and Q times the accumulated rotations the left singular vectors). One
// cluster per block, the block in shared memory, all blocks of a call in one launch.
//
// A QR-iteration SVD of such a block is some two hundred dependent launches with host decisions between
// them, whatever its size (a 40 x 40 block about 1.5 ms).
//   * The pivoted QR grades the columns that Jacobi sees: 7 to 9 sweeps where A itself takes 10
//     (flat spectrum) to 26 (decaying). Every CTA of a cluster does it for itself.
//   * A round of n / 2 disjoint pairs is three phases: dot products, rotation angles (one lane per
//     pair), rotations (one warp per pair). The CTAs share the rows of the rotated columns, swap
//     their parts of the dot products through distributed shared memory, and each finds the angles.
//   * All phases are bound by the FP64 pipe, where a warp instruction takes 64 cycles of a quarter of
//     the SM whatever its active lanes: reductions run over 4 or 8 lanes, and an angle is FP32 and
//     integer work where that will do, four warps sharing out the rest.
//   * Columns are kept as scale x stored column, so a rotation is one FMA per element (p - ta q,
//     q + tb p) instead of two operations; the scales are multiplied in once per sweep.
//   * The tangent of an angle needs few digits: it is taken in FP32, and the cosine that makes the
//     rotation orthogonal is refined to FP64 from it.
// Convergence: every pair's |<p, q>| <= sqrt(n) eps |p| |q|, so small singular vectors are as orthogonal
// as large ones. Columns that QR leaves below 1e-60 of the block's largest element count as that
// much. A block with a non-finite element is left to the caller.
// Measured against QR iteration: exact truncation of a chi = 128 two-site tensor (blocks up to 62 x 62)
// 5.58 -> 1.76 ms (3.79 ms with one CTA per block, a warp per reduction and the angles in FP64), an
// L = 32, chi = 64 two-site DMRG sweep (61 truncations) 208 -> 112 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "svd_small.hpp"

namespace mpsg {

namespace {

namespace cg = cooperative_groups;

// Smaller dimension. A 62 x 62 block takes 1.5 ms here and 5.3 ms by QR iteration, a 30 x 30 one 0.25 ms
// and 1.5 ms; larger ones outgrow an SM's shared memory and the lanes of a warp that finds the angles.
constexpr int kMaxCols = 64;
constexpr int kThreads = 512;
constexpr int kMaxSweeps = 30;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRows = 256;    // larger dimension (32 elements of a column per lane of eight)
constexpr int kCluster = 4;
// Columns up to which a launch gives each block one CTA: the angles, which every CTA finds, are then most
// of a round. The 61 truncations of an L = 32, chi = 64 sweep 15.3 ms, 15.8 ms with 32 here.
constexpr int kOneCta = 16;
constexpr double kFloor = 1e-60;
constexpr size_t kMaxSmem = 220 * 1024;

__host__ __device__ __forceinline__ int even_up(int n) { return n + (n & 1); }

// Lanes per pair in the dot products: all pairs on four warps.
__host__ __device__ __forceinline__ int pair_lanes(int np) { return np <= 16 ? 8 : 4; }

// Shared-memory layout of an m x n block (m >= n) in a cluster of C.
struct Layout {
  int ne, np;  // columns rounded up to an even number, pairs
  int nl;      // rows of R^T (and of V) per CTA: row i is row i / C of CTA i % C
  int ld, lh;  // strides of the rotated columns and of the QR factor (lanes on different banks)
  __host__ __device__ Layout(int m, int n, int C) {
    ne = even_up(n);
    np = ne / 2;
    nl = (n + C - 1) / C;
    const int gl = pair_lanes(np), g2 = 2 * gl;
    ld = 2 * nl + (gl + g2 - 2 * nl % g2) % g2;
    lh = m + (24 - m % 16) % 16;
  }
  size_t bytes(int n, int C) const {
    return sizeof(double) * ((size_t)ld * ne + (size_t)lh * n + 5 * (size_t)ne + 2 * (size_t)C * ne) +
           2 * sizeof(int) * (size_t)ne;
  }
};

// Column pair i of round r (circle method over an even number of columns).
__device__ __forceinline__ void pair_of(int i, int r, int ne, int& p, int& q) {
  if (i == 0) {
    p = r;
    q = ne - 1;
  } else {
    p = r + i;
    if (p >= ne - 1) p -= ne - 1;
    q = r - i;
    if (q < 0) q += ne - 1;
  }
}

// Biased exponent of x, and its significand in [1, 2) as FP32 (no FP64 instruction: a warp's takes 64
// cycles of its quarter of the pipe). 0 for zeros and subnormals.
__device__ __forceinline__ int split_float(double x, float& f) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  f = __int_as_float(0x3f800000 | (hi & 0xfffff) << 3 | (int)((unsigned)lo >> 29));
  return (hi >> 20) & 0x7ff;
}

// sign(z) / (|z| + sqrt(1 + z^2)), z = df / 2 g, to FP32's precision; eg, fg: g's parts
__device__ __forceinline__ double tangent(double df, double g, int eg, float fg) {
  float fd;
  const int ed = split_float(df, fd), D = ed - eg - 1;
  float t;
  int e = 0;
  if (ed == 0 || D < -60) {
    t = 1.f;
  } else if (D > 40) {  // 1 / 2 z
    t = __fdividef(fg, fd);
    e = eg - ed;
  } else {
    const float z = __fdividef(fd, fg) * __int_as_float((D + 127) << 23);
    t = __fdividef(1.f, z + sqrtf(fmaf(z, z, 1.f)));
  }
  const int bits = __float_as_int(t);
  e += (bits >> 23) + (1023 - 127);
  if (e <= 0) return 0.0;
  const int sign = (__double2hiint(df) ^ __double2hiint(g)) & 0x80000000;
  return __hiloint2double(sign | e << 20 | (bits & 0x7fffff) >> 3, bits << 29);
}

// The left singular vectors of columns `order[first], order[first + step], ..`: the reflectors on
// unit[c] (V[:, c]; 0), eight lanes a column, NR elements of it in each. z: the cluster's rotated columns.
template <int NR>
__device__ __forceinline__ void left_vectors(double* left, int m, int n, int rank, int first, int step,
                                             double* const* z, const Layout& y, const double* H,
                                             const double* fac, const double* unit, const int* col,
                                             const int* order) {
  const int t = threadIdx.x, l8 = t & 7, C = step;
  for (int j0 = 0; first + step * j0 < n; j0 += kThreads / 8) {
    const int jw = first + step * (j0 + (t >> 5) * 4), j = first + step * (j0 + (t >> 3));
    if (jw >= n) continue;  // whole warps
    const int c = order[j < n ? j : jw];
    double x[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = l8 + 8 * i;
      x[i] = r < n ? z[r % C][c * y.ld + y.nl + r / C] * unit[c] : 0.0;
    }
    for (int k = rank - 1; k >= 0; --k) {
      const double* v = H + col[k] * y.lh;
      double h[NR], s = 0.0;
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int r = l8 + 8 * i;
        h[i] = r >= k && r < m ? v[r] : 0.0;
        s = fma(h[i], x[i], s);
      }
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s *= -fac[k];
#pragma unroll
      for (int i = 0; i < NR; ++i) x[i] = fma(s, h[i], x[i]);
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = l8 + 8 * i;
      if (j < n && r < m) left[r + (int64_t)j * m] = x[i];
    }
  }
}

__global__ void __launch_bounds__(kThreads) jacobi_svd_kernel(
    const SmallSvdBlock* __restrict__ blocks, int C) {
  extern __shared__ double sm[];
  __shared__ int rotated, bad, pivot;
  __shared__ double wmax[kWarps];
  const auto cluster = cg::this_cluster();
  const int me = C > 1 ? (int)cluster.block_rank() : 0;
  const SmallSvdBlock B = blocks[blockIdx.x / C];
  const bool wide = B.M < B.N;  // then A^T is factorised
  const int m = wide ? B.N : B.M, n = wide ? B.M : B.N;
  const Layout y(m, n, C);
  const int ne = y.ne, np = y.np, nl = y.nl, ld = y.ld, lh = y.lh;
  double* Z = sm;               // ld x ne: this CTA's rows of W = R^T, below them its rows of V
  double* H = Z + ld * ne;      // lh x n: reflectors and R
  double* d = H + lh * n;       // squared norms
  double* sc = d + ne;          // column scales and their inverses
  double* isc = sc + ne;        // first the diagonal of R
  double* ta = isc + ne;        // rotation factors of a round's pairs
  double* tb = ta + np;
  double* fac = tb + np;        // reflector factors
  double* dots = fac + ne;      // [round parity][CTA][pair]: parts of the dot products
  double* norms = dots + C * ne;  // [CTA][column]: parts of the squared norms
  int* order = (int*)(norms + C * ne);
  int* col = order + ne;        // col[k]: column of A at position k
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  auto sync = [&] {
    if (C > 1) cluster.sync();
    else __syncthreads();
  };
  double* z[kCluster];
  for (int q = 0; q < kCluster; ++q) z[q] = C > 1 ? cluster.map_shared_rank(sm, q < C ? q : 0) : sm;
  if (t == 0) bad = 0;
  double mx = 0.0;
  int nonfinite = 0;
  for (int e = t; e < m * n; e += kThreads) {
    const int c = e / m, r = e - c * m;
    const double x = wide ? B.A[c + (int64_t)r * B.M] : B.A[e];
    H[c * lh + r] = x;
    nonfinite |= (__double2hiint(x) & 0x7ff00000) == 0x7ff00000;
    mx = fmax(mx, fabs(x));
  }
  for (int e = t; e < ld * ne; e += kThreads) {
    const int c = e / ld, r = e - c * ld - nl;
    Z[e] = r >= 0 && r < nl && r * C + me == c && c < n ? 1.0 : 0.0;
  }
  for (int j = t; j < n; j += kThreads) col[j] = j;
  for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) wmax[w] = mx;
  __syncthreads();
  if (nonfinite) bad = 1;
  mx = 0.0;
  for (int i = 0; i < kWarps; ++i) mx = fmax(mx, wmax[i]);
  const bool zero = mx == 0.0;
  const int ex = zero ? 0 : ((__double2hiint(mx) >> 20) & 0x7ff) - 1023;
  __syncthreads();
  if (bad || ex < -900 || ex > 900) {  // the same in every CTA of the cluster
    if (t == 0) *B.info = 1;
    return;
  }
  // scale by the power of two that brings the largest element to about 1; squared column norms
  const double down = __hiloint2double((1023 - ex) << 20, 0);
  for (int c = w; c < n; c += kWarps) {
    double s = 0.0;
    for (int r = lane; r < m; r += 32) {
      const double x = H[c * lh + r] * down;
      H[c * lh + r] = x;
      s = fma(x, x, s);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) d[c] = s;
  }
  __syncthreads();
  // QR: reflector k = I - fac v v^T on the largest remaining column (v in its place, its R element in
  // isc[k]); the update of each other column (eight lanes each) also takes the norm of what remains
  int rank = n;
  const int l8 = lane & 7;
  for (int k = 0; k < n; ++k) {
    if (w == 0) {
      unsigned best = 0;
      int at = k;
      for (int j = k + lane; j < n; j += 32) {  // norm^2 >= 1e-120: compare by the high word
        const unsigned h = (unsigned)__double2hiint(d[col[j]]) + 1;
        if (h > best) {
          best = h;
          at = j;
        }
      }
      const unsigned top = __reduce_max_sync(0xffffffffu, best);
      const int from = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
      at = __shfl_sync(0xffffffffu, at, from);
      if (lane == 0) {
        const int c = col[at];
        col[at] = col[k];
        col[k] = c;
        const double nn = d[c];
        if (nn < kFloor * kFloor) {
          pivot = -1;
        } else {
          const double alpha = H[c * lh + k], s = sqrt(nn), beta = alpha > 0.0 ? -s : s;
          pivot = c;
          isc[k] = beta;
          H[c * lh + k] = alpha - beta;
          fac[k] = 1.0 / (beta * (beta - alpha));  // 2 / v^T v
        }
      }
    }
    __syncthreads();
    if (pivot < 0) {  // all that remains is below the floor
      rank = k;
      break;
    }
    const double* v = H + pivot * lh;
    const double f = -fac[k];
    for (int j0 = k + 1 + 4 * w; j0 < n; j0 += 4 * kWarps) {
      const int j = j0 + (lane >> 3), end = j < n ? m : 0;
      double* x = H + col[j < n ? j : k] * lh;
      double s = 0.0, q = 0.0;
      for (int r = k + l8; r < end; r += 8) s = fma(v[r], x[r], s);
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s *= f;
      for (int r = k + l8; r < end; r += 8) {
        const double u = fma(s, v[r], x[r]);
        x[r] = u;
        if (r > k) q = fma(u, u, q);
      }
      for (int o = 4; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (l8 == 0 && j < n) d[col[j]] = q;
    }
    __syncthreads();
  }
  // W = R^T, this CTA's rows
  for (int e = t; e < n * nl; e += kThreads) {
    const int k = e / nl, i = e - k * nl, j = i * C + me;  // R(k, j), k <= j
    if (j >= n) continue;
    if (k == j) Z[k * ld + i] = k < rank ? isc[k] : kFloor;
    else if (k < j && k < rank) Z[k * ld + i] = H[col[j] * lh + k];
  }
  // a pair is rotated when 2 log2 |g| > log2 |p|^2 + log2 |q|^2 + log2 (n eps^2)
  const float tol = __log2f((float)(n < 10 ? 10 : n)) - 104.f;
  const int gl = pair_lanes(np), gi = t / gl, gk = t & (gl - 1);
  bool done = false;
  sync();  // every CTA of the cluster runs before one writes to another
  for (int sweep = 0; sweep < kMaxSweeps && !done; ++sweep) {
    __syncthreads();
    if (t == 0) rotated = 0;
    // multiply the scales in, then the norms
    if (sweep)
      for (int c = w; c < n; c += kWarps) {
        const double s = sc[c];
        for (int r = lane; r < 2 * nl; r += 32) Z[c * ld + r] *= s;
      }
    __syncthreads();
    {
      static_assert(kThreads / 8 >= kMaxCols, "eight lanes a column");
      const int c = t >> 3, end = c < n ? nl : 0;
      double s = 0.0;
      for (int r = l8; r < end; r += 8) s = fma(Z[c * ld + r], Z[c * ld + r], s);
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (c < ne && l8 < C) z[l8][norms - sm + me * ne + c] = s;
    }
    sync();
    if (t < ne) {
      double s = norms[t];
      for (int q = 1; q < C; ++q) s += norms[q * ne + t];
      d[t] = s;
      sc[t] = isc[t] = 1.0;
      if (t < n && !(s > 1e-290)) bad = 1;
    }
    __syncthreads();
    if (bad) break;
    for (int r = 0; r < ne - 1; ++r) {
      const double* part = dots + (r & 1) * C * np;
      if (w < 4) {
        double s = 0.0, s1 = 0.0;
        if (gi < np) {
          int p, q;
          pair_of(gi, r, ne, p, q);
          const double *wp = Z + p * ld, *wq = Z + q * ld;
          int k = gk;
          for (; k + gl < nl; k += 2 * gl) {
            s = fma(wp[k], wq[k], s);
            s1 = fma(wp[k + gl], wq[k + gl], s1);
          }
          if (k < nl) s = fma(wp[k], wq[k], s);
        }
        s += s1;
        for (int o = gl >> 1; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (gi < np && gk < C) z[gk][part - sm + me * np + gi] = s;
      }
      sync();
      if (w < 4) {  // all four find the cosine; each writes its part of the results
        const bool in = lane < np;
        int p = 0, q = 0;
        double dp, dq, sp, sq, ip, iq, g;
        if (in) {
          pair_of(lane, r, ne, p, q);
          dp = d[p], dq = d[q], sp = sc[p], sq = sc[q], ip = isc[p], iq = isc[q];
          g = part[lane];
          for (int c = 1; c < C; ++c) g += part[c * np + lane];
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");  // all have read what some write
        if (in) {
          g = g * sp * sq;
          float fp, fq, fg;
          const int ep = split_float(dp, fp), eq = split_float(dq, fq), eg = split_float(g, fg);
          const bool on = ep && eq && eg &&
                          (2.f * __log2f(fg) - __log2f(fp) - __log2f(fq)) +
                                  (float)(2 * eg - ep - eq) > tol;
          if (!on) {
            if (w == 0) ta[lane] = 0.0;
          } else {
            const double tt = tangent(dq - dp, g, eg, fg);
            if (w == 2) {
              const double dp1 = fma(-tt, g, dp), dq1 = fma(tt, g, dq);
              d[p] = __double2hiint(dp1) < 0 ? 0.0 : dp1;
              d[q] = __double2hiint(dq1) < 0 ? 0.0 : dq1;
              rotated = 1;
            }
            if (w == 0) {
              ta[lane] = tt * (sq * ip);
            } else if (w == 1) {
              tb[lane] = tt * (sp * iq);
            } else {
              // 1 / sqrt(1 + tan^2) and its inverse: FP32 seed, one step of third order
              const double u = fma(tt, tt, 1.0), c0 = (double)rsqrtf((float)u);
              const double res = fma(-u * c0, c0, 1.0), c = fma(c0 * res, fma(0.375, res, 0.5), c0);
              if (w == 2) {
                sc[p] = sp * c;
                sc[q] = sq * c;
              } else {
                const double ic = c * u;
                isc[p] = ip * ic;
                isc[q] = iq * ic;
              }
            }
          }
        }
      }
      __syncthreads();
      for (int i = w; i < np; i += kWarps) {
        const double a = ta[i], b = tb[i];
        if (a == 0.0) continue;
        int p, q;
        pair_of(i, r, ne, p, q);
        double *zp = Z + p * ld, *zq = Z + q * ld;
#pragma unroll 4
        for (int k = lane; k < 2 * nl; k += 32) {
          const double x = zp[k], x1 = zq[k];
          zp[k] = fma(-a, x1, x);
          zq[k] = fma(b, x, x1);
        }
      }
      __syncthreads();
    }
    done = rotated == 0;
  }
  sync();  // the columns are read across the cluster below
  if (!done) {
    if (t == 0) *B.info = 1;
    return;
  }
  // The rotations' rounding has moved the norms of V's columns by some eps: squared norms again, and the
  // factors (ta) that bring them, and with them the singular values, back.
  {
    const int c = t >> 3, end = c < n ? nl : 0;
    const double* v = Z + c * ld + nl;
    double s = 0.0;
    for (int r = l8; r < end; r += 8) s = fma(v[r], v[r], s);
    for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (c < ne && l8 < C) z[l8][norms - sm + me * ne + c] = s;
  }
  sync();
  // singular values (d holds the squared norms of the last, rotation-free sweep), descending order
  if (t < n) {
    double v = norms[t];
    for (int q = 1; q < C; ++q) v += norms[q * ne + t];
    ta[t] = fma(-0.5, v, 1.5);
    const double s = sqrt(d[t]);
    isc[t] = 1.0 / s;
    sc[t] = s * ta[t] * (zero ? 0.0 : __hiloint2double((1023 + ex) << 20, 0));
  }
  __syncthreads();
  if (t < n) {
    int at = 0;
    for (int i = 0; i < n; ++i) at += sc[i] > sc[t] || (sc[i] == sc[t] && i < t);
    order[at] = t;
  }
  __syncthreads();
  double* left = wide ? B.V : B.U;
  double* right = wide ? B.U : B.V;
  if (me == 0 && t < n) B.S[t] = sc[order[t]];
  for (int e = t; e < n * nl; e += kThreads) {
    const int j = e / nl, i = e - j * nl, c = order[j];
    if (i * C + me < n) right[col[i * C + me] + (int64_t)j * n] = Z[c * ld + i] * isc[c];
  }
  if (m <= 64) left_vectors<8>(left, m, n, rank, me, C, z, y, H, fac, ta, col, order);
  else if (m <= 128) left_vectors<16>(left, m, n, rank, me, C, z, y, H, fac, ta, col, order);
  else left_vectors<32>(left, m, n, rank, me, C, z, y, H, fac, ta, col, order);
  if (C > 1) cluster.sync();  // its columns may still be read
}

}  // namespace

bool small_svd_fits(int64_t M, int64_t N) {
  const int64_t n = std::min(M, N), m = std::max(M, N);
  return n >= 1 && n <= kMaxCols && m <= kMaxRows;
}

void launch_small_svd(Context* ctx, const std::vector<SmallSvdBlock>& blocks) {
  if (blocks.empty()) return;
  static std::once_flag smem_set[kMaxDevices];
  set_smem_limit_once(ctx, smem_set, jacobi_svd_kernel, (int)kMaxSmem);
  std::vector<SmallSvdBlock> sorted(blocks);  // the largest first
  std::stable_sort(sorted.begin(), sorted.end(), [](const SmallSvdBlock& a, const SmallSvdBlock& b) {
    return std::min(a.M, a.N) > std::min(b.M, b.N);
  });
  // Clusters while there are SMs for all blocks, unless the angles are most of a round anyway.
  const int64_t n = std::min(sorted[0].M, sorted[0].N);
  int C = n > kOneCta ? kCluster : 1;
  while (C > 1 && (int64_t)sorted.size() * C > ctx->num_sms) C /= 2;
  size_t smem = 0;
  for (const SmallSvdBlock& b : sorted) {
    const int k = std::min(b.M, b.N);
    smem = std::max(smem, Layout(std::max(b.M, b.N), k, C).bytes(k, C));
  }
  TableImage img;
  img.add(sorted);
  unsigned char* d = img.upload(ctx->stream);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sorted.size() * (unsigned)C);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  MPSG_CUDA(cudaLaunchKernelEx(&cfg, jacobi_svd_kernel, (const SmallSvdBlock*)d, C));
  ctx->kernel_launches++;
  MPSG_CUDA(cudaFreeAsync(d, ctx->stream));
}

}  // namespace mpsg
