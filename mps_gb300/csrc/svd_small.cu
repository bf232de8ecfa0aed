// Thin SVD of small blocks: column-pivoted Householder QR, A P = Q R, then one-sided Jacobi on R^T (plane
// rotations of column pairs until all columns are orthogonal: their norms are the singular values, the
// normalised columns the right and Q times the accumulated rotations the left singular vectors). One
// CTA per block, the block in shared memory, all blocks of a call in one launch.
//
// A QR-iteration SVD of such a block is some two hundred dependent launches with host decisions between
// them, whatever its size (a 40 x 40 block about 1.5 ms).
//   * The pivoted QR grades the columns that Jacobi sees: 7 to 9 sweeps where A itself takes 10
//     (flat spectrum) to 26 (decaying).
//   * A round of n / 2 disjoint pairs is three phases: dot products (eight lanes per pair), rotation
//     angles (one lane per pair: scalar FP64 work would cost every other lane of a warp its slot on a
//     pipe of 2 FMAs per cycle), rotations (one warp per pair).
//   * Columns are kept as scale x stored column, so a rotation is one FMA per element (p - ta q,
//     q + tb p) instead of two operations; the scales are multiplied in once per sweep.
//   * The tangent of an angle needs few digits: it is taken in FP32, and the cosine that makes the
//     rotation orthogonal is refined to FP64 from it.
// Convergence: every pair's |<p, q>| <= sqrt(n) eps |p| |q|, so small singular vectors are as orthogonal
// as large ones. Columns that QR leaves below 1e-60 of the block's largest element count as that
// much. A block with a non-finite element is left to the caller.
// Measured against QR iteration: exact truncation of a chi = 128 two-site tensor (blocks up to 63 x 63)
// 5.58 -> 3.79 ms, an L = 32, chi = 64 two-site DMRG sweep (61 truncations) 208 -> 120 ms.
#include <algorithm>

#include "svd_small.hpp"

namespace mpsg {

namespace {

// Smaller dimension. A 63 x 63 block takes 3.5 ms here and 5.3 ms by QR iteration, a 30 x 30 one 0.4 ms
// and 1.5 ms; larger ones outgrow one SM's shared memory and its FP64 pipe.
constexpr int kMaxCols = 64;
constexpr int kThreads = 512;
constexpr int kMaxSweeps = 30;
constexpr size_t kMaxSmem = 200 * 1024;

__host__ __device__ __forceinline__ int even_up(int n) { return n + (n & 1); }

constexpr int kMaxRows = 256;    // larger dimension (eight elements of a column per lane)
constexpr double kFloor = 1e-60;

// W, V (n x ne), the QR factor (m x n), five vectors of ne, two index vectors
size_t smem_bytes(int m, int n) {
  const int ne = even_up(n);
  return sizeof(double) * ((size_t)m * n + 2 * (size_t)n * ne + 5 * (size_t)ne) +
         2 * sizeof(int) * (size_t)ne;
}

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

__global__ void __launch_bounds__(kThreads) jacobi_svd_kernel(
    const SmallSvdBlock* __restrict__ blocks) {
  extern __shared__ double sm[];
  __shared__ int rotated, bad, pivot;
  __shared__ double wmax[kThreads / 32], refl[2];
  const SmallSvdBlock B = blocks[blockIdx.x];
  const bool wide = B.M < B.N;  // then A^T is factorised
  const int m = wide ? B.N : B.M, n = wide ? B.M : B.N, ne = even_up(n), np = ne / 2;
  double* W = sm;               // n x ne
  double* V = W + n * ne;       // n x ne
  double* H = V + n * ne;       // m x n: reflectors and R
  double* d = H + m * n;        // squared norms
  double* sc = d + ne;          // column scales and their inverses; first reflector factors
  double* isc = sc + ne;        // first diagonal of R
  double* ta = isc + ne;        // rotation factors of a round's pairs (first: their dot products)
  double* tb = ta + np;
  double* fac = tb + np;        // reflector factors
  int* order = (int*)(fac + ne);
  int* col = order + ne;        // col[k]: column of A at position k
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  constexpr int kWarps = kThreads / 32;
  if (t == 0) bad = 0;
  double mx = 0.0;
  int nonfinite = 0;
  for (int e = t; e < m * n; e += kThreads) {
    const int c = e / m, r = e - c * m;
    const double x = wide ? B.A[c + (int64_t)r * B.M] : B.A[e];
    H[e] = x;
    nonfinite |= (__double2hiint(x) & 0x7ff00000) == 0x7ff00000;
    mx = fmax(mx, fabs(x));
  }
  for (int e = t; e < n * ne; e += kThreads) {
    V[e] = e / n == e % n ? 1.0 : 0.0;
    W[e] = 0.0;
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
  if (bad || ex < -900 || ex > 900) {
    if (t == 0) *B.info = 1;
    return;
  }
  // scale by the power of two that brings the largest element to about 1; squared column norms
  const double down = __hiloint2double((1023 - ex) << 20, 0);
  for (int c = w; c < n; c += kWarps) {
    double s = 0.0;
    for (int r = lane; r < m; r += 32) {
      const double x = H[c * m + r] * down;
      H[c * m + r] = x;
      s = fma(x, x, s);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) d[c] = s;
  }
  __syncthreads();
  // QR: reflector k = I - fac v v^T on the largest remaining column (v in its place, its R element in
  // isc[k]); the update of each other column also takes the norm of what remains of it
  int rank = n;
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
          const double alpha = H[c * m + k], s = sqrt(nn), beta = alpha > 0.0 ? -s : s;
          pivot = c;
          isc[k] = beta;
          H[c * m + k] = alpha - beta;
          fac[k] = 1.0 / (beta * (beta - alpha));  // 2 / v^T v
        }
      }
    }
    __syncthreads();
    if (pivot < 0) {  // all that remains is below the floor
      rank = k;
      break;
    }
    const double* v = H + pivot * m;
    const double f = fac[k];
    for (int j = k + 1 + w; j < n; j += kWarps) {
      double* y = H + col[j] * m;
      double s = 0.0;
      for (int r = k + lane; r < m; r += 32) s = fma(v[r], y[r], s);
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s *= f;
      double q = 0.0;
      for (int r = k + lane; r < m; r += 32) {
        const double x = fma(-s, v[r], y[r]);
        y[r] = x;
        if (r > k) q = fma(x, x, q);
      }
      for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (lane == 0) d[col[j]] = q;
    }
    __syncthreads();
  }
  // W = R^T
  for (int e = t; e < n * n; e += kThreads) {
    const int j = e / n, k = e - j * n;  // R(k, j), k <= j
    if (k == j) W[k * n + j] = k < rank ? isc[k] : kFloor;
    else if (k < j && k < rank) W[k * n + j] = H[col[j] * m + k];
  }
  __syncthreads();
  for (int j = t; j < ne; j += kThreads) sc[j] = isc[j] = 1.0;
  const double tol = 4.93e-32 * (n < 10 ? 10 : n);
  const int g8 = t >> 3, l8 = t & 7;  // groups of eight lanes
  bool done = false;
  for (int sweep = 0; sweep < kMaxSweeps && !done; ++sweep) {
    __syncthreads();
    if (t == 0) rotated = 0;
    // multiply the scales in, then the norms
    if (sweep)
      for (int c = w; c < n; c += kWarps) {
        const double s = sc[c];
        for (int r = lane; r < n; r += 32) {
          W[c * n + r] *= s;
          V[c * n + r] *= s;
        }
      }
    __syncthreads();
    for (int c0 = 0; c0 < ne; c0 += kThreads / 8) {  // whole warps take part in the shuffles
      const int c = c0 + g8;
      double s = 0.0;
      if (c < ne)
        for (int r = l8; r < n; r += 8) s = fma(W[c * n + r], W[c * n + r], s);
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, 8);
      if (c < ne && l8 == 0) {
        d[c] = s;
        sc[c] = isc[c] = 1.0;
        if (c < n && !(s > 1e-290)) bad = 1;
      }
    }
    __syncthreads();
    if (bad) break;
    for (int r = 0; r < ne - 1; ++r) {
      for (int i0 = 0; i0 < np; i0 += kThreads / 8) {
        const int i = i0 + g8;
        double s = 0.0;
        int p = 0, q = 0;
        if (i < np) {
          pair_of(i, r, ne, p, q);
          for (int k = l8; k < n; k += 8) s = fma(W[p * n + k], W[q * n + k], s);
        }
        for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, 8);
        if (i < np && l8 == 0) ta[i] = s;
      }
      __syncthreads();
      if (t < np) {
        int p, q;
        pair_of(t, r, ne, p, q);
        const double dp = d[p], dq = d[q], g = ta[t] * sc[p] * sc[q];
        double a = 0.0, b = 0.0;
        if (g * g > tol * (dp * dq)) {
          // tan = sign(z) / (|z| + sqrt(1 + z^2)), z = (dq - dp) / 2 g, relative to the larger norm
          const int e = __double2hiint(fmax(dp, dq)) & 0x7ff00000;
          const double by = __hiloint2double(0x7fe00000 - e, 0), df = (dq - dp) * by, h = g * by;
          double tt;
          if (fabs(h) > 1e-30) {
            const float zf = __fdividef(0.5f * (float)df, (float)h), za = fabsf(zf);
            const float tf = za > 1e9f ? __fdividef(0.5f, za)
                                       : __fdividef(1.f, za + sqrtf(fmaf(za, za, 1.f)));
            tt = zf < 0.f ? -(double)tf : (double)tf;
          } else {
            tt = df != 0.0 ? h / df : 1.0;
          }
          const double u = fma(tt, tt, 1.0);
          double c = (double)rsqrtf((float)u);
          c = c * fma(-0.5 * u * c, c, 1.5);
          c = c * fma(-0.5 * u * c, c, 1.5);
          a = tt * sc[q] * isc[p];
          b = tt * sc[p] * isc[q];
          sc[p] *= c;
          sc[q] *= c;
          const double ic = c * u;  // 1 / c
          isc[p] *= ic;
          isc[q] *= ic;
          const double c2 = c * c, x = 2.0 * tt * g, t2 = tt * tt;
          d[p] = fmax(c2 * (dp - x + t2 * dq), 0.0);
          d[q] = fmax(c2 * (dq + x + t2 * dp), 0.0);
          rotated = 1;
        }
        ta[t] = a;
        tb[t] = b;
      }
      __syncthreads();
      for (int i = w; i < np; i += kWarps) {
        const double a = ta[i], b = tb[i];
        if (a == 0.0) continue;
        int p, q;
        pair_of(i, r, ne, p, q);
        double *wp = W + p * n, *wq = W + q * n, *vp = V + p * n, *vq = V + q * n;
        for (int k = lane; k < n; k += 32) {
          const double x = wp[k], y = wq[k], x1 = vp[k], y1 = vq[k];
          wp[k] = fma(-a, y, x);
          wq[k] = fma(b, x, y);
          vp[k] = fma(-a, y1, x1);
          vq[k] = fma(b, x1, y1);
        }
      }
      __syncthreads();
    }
    done = rotated == 0;
  }
  __syncthreads();
  if (!done) {
    if (t == 0) *B.info = 1;
    return;
  }
  // descending order (d holds the squared norms of the last, rotation-free sweep)
  for (int j = t; j < n; j += kThreads) {
    int at = 0;
    for (int i = 0; i < n; ++i) at += d[i] > d[j] || (d[i] == d[j] && i < j);
    order[at] = j;
  }
  __syncthreads();
  double* left = wide ? B.V : B.U;
  double* right = wide ? B.U : B.V;
  const double up = zero ? 0.0 : __hiloint2double((1023 + ex) << 20, 0);
  for (int j = w; j < n; j += kWarps) {
    const int c = order[j];
    const double s = sqrt(d[c]), inv = 1.0 / s;
    if (lane == 0) B.S[j] = s * up;
    for (int r = lane; r < n; r += 32) right[col[r] + (int64_t)j * n] = W[c * n + r] * inv;
    // left vector: the reflectors on (V[:, c]; 0), eight elements a lane
    double x[kMaxRows / 32];
#pragma unroll
    for (int i = 0; i < kMaxRows / 32; ++i) {
      const int r = lane + 32 * i;
      x[i] = r < n ? V[c * n + r] : 0.0;
    }
    for (int k = rank - 1; k >= 0; --k) {
      const double* v = H + col[k] * m;
      double s0 = 0.0;
#pragma unroll
      for (int i = 0; i < kMaxRows / 32; ++i) {
        const int r = lane + 32 * i;
        if (r >= k && r < m) s0 = fma(v[r], x[i], s0);
      }
      for (int o = 16; o; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s0 *= fac[k];
#pragma unroll
      for (int i = 0; i < kMaxRows / 32; ++i) {
        const int r = lane + 32 * i;
        if (r >= k && r < m) x[i] = fma(-s0, v[r], x[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < kMaxRows / 32; ++i) {
      const int r = lane + 32 * i;
      if (r < m) left[r + (int64_t)j * m] = x[i];
    }
  }
}

}  // namespace

bool small_svd_fits(int64_t M, int64_t N) {
  const int64_t n = std::min(M, N), m = std::max(M, N);
  return n >= 1 && n <= kMaxCols && m <= kMaxRows && smem_bytes((int)m, (int)n) <= kMaxSmem;
}

void launch_small_svd(Context* ctx, const std::vector<SmallSvdBlock>& blocks) {
  if (blocks.empty()) return;
  static std::once_flag smem_set[kMaxDevices];
  set_smem_limit_once(ctx, smem_set, jacobi_svd_kernel, (int)kMaxSmem);
  std::vector<SmallSvdBlock> sorted(blocks);  // the largest first
  std::stable_sort(sorted.begin(), sorted.end(), [](const SmallSvdBlock& a, const SmallSvdBlock& b) {
    return std::min(a.M, a.N) > std::min(b.M, b.N);
  });
  size_t smem = 0;
  for (const SmallSvdBlock& b : sorted)
    smem = std::max(smem, smem_bytes(std::max(b.M, b.N), std::min(b.M, b.N)));
  TableImage img;
  img.add(sorted);
  unsigned char* d = img.upload(ctx->stream);
  jacobi_svd_kernel<<<(unsigned)sorted.size(), kThreads, smem, ctx->stream>>>((SmallSvdBlock*)d);
  MPSG_CUDA(cudaGetLastError());
  ctx->kernel_launches++;
  MPSG_CUDA(cudaFreeAsync(d, ctx->stream));
}

}  // namespace mpsg
