// Thick-restart Lanczos on device-resident tensors (the KrylovKit.eigsolve call of
// src/dmrg.jl:77-82).  Krylov vectors, reorthogonalisation dot products and vector updates are
// FP64 kernels on the context stream; the host keeps only the small projected matrix.
//
// Measured, ground-state solve at chi = 256 (19 products, krylovdim 5, 8 cycles): 4.6 ms with a dozen
// launches and one host synchronisation per step and the projected matrix decomposed by one warp
// (112 us a cycle), 2.6 ms with one launch per step (21 us) and the host kLag steps behind.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "linalg.hpp"

namespace mpsg {

void small_eigh(int n, const double* A, double* evals, double* evecs) {
  std::vector<double> a(A, A + n * n), v(n * n, 0.0);
  for (int i = 0; i < n; ++i) v[i * n + i] = 1.0;
  auto at = [&](int i, int j) -> double& { return a[i + n * j]; };
  for (int sweep = 0; sweep < 100; ++sweep) {
    double off = 0.0, diag = 0.0;
    for (int j = 0; j < n; ++j)
      for (int i = 0; i < n; ++i) (i == j ? diag : off) += at(i, j) * at(i, j);
    if (off <= 1e-32 * std::max(diag, 1e-300)) break;
    for (int p = 0; p < n - 1; ++p)
      for (int q = p + 1; q < n; ++q) {
        double apq = at(p, q);
        if (apq == 0.0) continue;
        double theta = (at(q, q) - at(p, p)) / (2.0 * apq);
        double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < n; ++k) {  // rotate columns p, q
          double akp = at(k, p), akq = at(k, q);
          at(k, p) = c * akp - s * akq;
          at(k, q) = s * akp + c * akq;
        }
        for (int k = 0; k < n; ++k) {  // rotate rows p, q
          double apk = at(p, k), aqk = at(q, k);
          at(p, k) = c * apk - s * aqk;
          at(q, k) = s * apk + c * aqk;
        }
        for (int k = 0; k < n; ++k) {
          double vkp = v[k + n * p], vkq = v[k + n * q];
          v[k + n * p] = c * vkp - s * vkq;
          v[k + n * q] = s * vkp + c * vkq;
        }
      }
  }
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  std::sort(order.begin(), order.end(), [&](int x, int y) {  // (an order of all values: NaN last)
    return at(x, x) < at(y, y) || (std::isnan(at(y, y)) && !std::isnan(at(x, x)));
  });
  for (int i = 0; i < n; ++i) {
    evals[i] = at(order[i], order[i]);
    for (int k = 0; k < n; ++k) evecs[k + n * i] = v[k + n * order[i]];
  }
}

namespace {

constexpr int kMaxKrylov = 32;
constexpr int kVecThreads = 256;
constexpr long long kBarrierCycles = 4000000000LL;  // about 2 s at the maximum SM clock

// Short vectors are left to one cluster of so many blocks, which meets at its hardware barrier (0.4 us
// against about 2 us at a counter) and takes up to kClusterRows elements per thread: from about there
// on, the FP64 pipes of more SMs save more than the barriers cost. chi = 64 DMRG sweep of 32 sites
// 91.0 ms at the counter, 88.1 ms so.
constexpr int kClusterBlocks = 8, kClusterRows = 3;

// The vector part of a Lanczos solve runs as cooperative launches whose blocks meet at a counter in
// device memory: one launch per Krylov step instead of a dozen (dots, sums, coefficients,
// updates, twice, then the norm and the scaling), each of which would read the vectors again and
// wait for the one before.
struct GridBarrier {
  unsigned* count;   // arrivals since the solve began
  unsigned target;   // arrivals after the first barrier of this launch
  int* err;
};

// Barrier number i of the launch. Bounded: on expiry an error code is recorded and the block goes on.
__device__ __forceinline__ void grid_barrier(const GridBarrier& b, int i) {
  if (gridDim.x == 1) {
    __syncthreads();
    return;
  }
  if (b.count == nullptr) {  // the grid is one cluster
    cooperative_groups::this_cluster().sync();
    return;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(b.count, 1u);
    const unsigned target = b.target + (unsigned)i * gridDim.x;
    const long long t0 = clock64();
    while ((int)(*(volatile unsigned*)b.count - target) < 0)
      if (clock64() - t0 > kBarrierCycles) {
        record_wait(b.err, 1);
        break;
      }
    __threadfence();
  }
  __syncthreads();
}

// Sum of every thread's v[0..n) over the block into part[j * gridDim.x + blockIdx.x] (v is used up). The
// lanes halve the list as they go: N / 2 additions, N / 4, .., one a step, instead of five per value.
template <int N>
__device__ __forceinline__ void block_partials(double (&v)[N], int n, double* part) {
  __shared__ double sh[kVecThreads / 32][N];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int j0 = 0;  // the value this lane holds a part of
#pragma unroll
  for (int o = 16, m = N / 2; o; o >>= 1, m >>= 1) {
    if (m == 0) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      continue;
    }
    const bool upper = (lane & o) != 0;
    if (upper) j0 += m;
#pragma unroll
    for (int j = 0; j < m; ++j) {
      const double keep = upper ? v[j + m] : v[j], give = upper ? v[j] : v[j + m];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  constexpr int kSame = N >= 32 ? 1 : 32 / N;  // lanes that hold one value
  if ((lane & (kSame - 1)) == 0) sh[w][j0] = v[0];
  __syncthreads();
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double x = 0.0;
    for (int i = 0; i < kVecThreads / 32; ++i) x += sh[i][j];
    part[(int64_t)j * gridDim.x + blockIdx.x] = x;
  }
  __syncthreads();
}

// out[j] = sum of part[j][*] over the blocks, in every block alike (a warp per j, fixed order).
__device__ __forceinline__ void sum_partials(const double* part, int n, double* out) {
  const int lane = threadIdx.x & 31;
  for (int j = threadIdx.x >> 5; j < n; j += kVecThreads / 32) {
    double x = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32)
      x += __ldcg(part + (int64_t)j * gridDim.x + b);
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) out[j] = x;
  }
  __syncthreads();
}

struct StepArgs {
  const double* V[kMaxKrylov];
  double* w;
  double* next;      // w normalised: the next basis vector
  double* part;      // 3 areas of K x gridDim.x partial sums
  double* out;       // [0] the projection on the newest vector, [1] the norm of what is left
  int K;
  int64_t n;
  GridBarrier bar;
};

// Classical Gram-Schmidt of w against V[0..K), twice, and the norm of the rest. The second pass'
// dot products are taken while the first pass' update has w and V in registers, so V is read
// three times in all. Bound by HBM or L2 (3 (K + 1) x 8 bytes per element) for long vectors, by the
// three barriers (about 2 us each) for short ones.
template <int KT>
__global__ void __launch_bounds__(kVecThreads) krylov_step_kernel(const __grid_constant__ StepArgs a) {
  __shared__ double c[KT];
  const int K = a.K;
  const int64_t n = a.n, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t area = (int64_t)K * gridDim.x;
  double d[KT];
#pragma unroll
  for (int j = 0; j < KT; ++j) d[j] = 0.0;
  for (int64_t e = first; e < n; e += stride) {
    const double w = a.w[e];
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < K) d[j] = fma(a.V[j][e], w, d[j]);
  }
  block_partials(d, K, a.part);
  grid_barrier(a.bar, 0);
  sum_partials(a.part, K, c);
  const double alpha1 = c[K - 1];
#pragma unroll
  for (int j = 0; j < KT; ++j) d[j] = 0.0;
  for (int64_t e = first; e < n; e += stride) {
    double v[KT], w = a.w[e];
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < K) {
        v[j] = a.V[j][e];
        w = fma(-c[j], v[j], w);
      }
    a.w[e] = w;
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < K) d[j] = fma(v[j], w, d[j]);
  }
  block_partials(d, K, a.part + area);
  grid_barrier(a.bar, 1);
  sum_partials(a.part + area, K, c);
  double s[1] = {0.0};
  for (int64_t e = first; e < n; e += stride) {
    double w = a.w[e];
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < K) w = fma(-c[j], a.V[j][e], w);
    a.w[e] = w;
    s[0] = fma(w, w, s[0]);
  }
  const double alpha = alpha1 + c[K - 1];
  block_partials(s, 1, a.part + 2 * area);
  grid_barrier(a.bar, 2);
  sum_partials(a.part + 2 * area, 1, c);
  const double beta = sqrt(c[0]);
  const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
  for (int64_t e = first; e < n; e += stride) a.next[e] = inv * a.w[e];
  if (first == 0) {
    a.out[0] = alpha;
    a.out[1] = beta;
  }
}

struct CombineArgs {
  const double* V[kMaxKrylov];
  double c[kMaxKrylov];
  double* x;
  double* part;
  double* out;       // the norm of the combination
  int K;
  int64_t n;
  GridBarrier bar;
};

// x = sum_j c_j V_j divided by its norm (K = 1, c = 1: a vector normalised).
__global__ void __launch_bounds__(kVecThreads) krylov_combine_kernel(
    const __grid_constant__ CombineArgs a) {
  __shared__ double c[1];
  const int64_t n = a.n, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double s[1] = {0.0};
  for (int64_t e = first; e < n; e += stride) {
    double x = 0.0;
    for (int j = 0; j < a.K; ++j) x = fma(a.c[j], a.V[j][e], x);
    a.x[e] = x;
    s[0] = fma(x, x, s[0]);
  }
  block_partials(s, 1, a.part);
  grid_barrier(a.bar, 0);
  sum_partials(a.part, 1, c);
  const double norm = sqrt(c[0]);
  const double inv = norm > 0.0 ? 1.0 / norm : 0.0;
  for (int64_t e = first; e < n; e += stride) a.x[e] *= inv;
  if (first == 0) *a.out = norm;
}

struct RestartArgs {
  double* V[kMaxKrylov];
  double U[kMaxKrylov * kMaxKrylov];  // [kept vector][old vector]
  int K, keep;
  int64_t n;
};

// V_i <- sum_j U(j, i) V_j for i < keep, in place: a thread reads its element of every vector before
// it writes any.
template <int KT>
__global__ void __launch_bounds__(kVecThreads) krylov_restart_kernel(
    const __grid_constant__ RestartArgs a) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < a.n;
       e += (int64_t)gridDim.x * blockDim.x) {
    double v[KT];
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < a.K) v[j] = a.V[j][e];
    for (int i = 0; i < a.keep; ++i) {
      double x = 0.0;
#pragma unroll
      for (int j = 0; j < KT; ++j)
        if (j < a.K) x = fma(a.U[i * a.K + j], v[j], x);
      a.V[i][e] = x;
    }
  }
}

template <class Args>
void launch_clustered(void (*kernel)(Args), dim3 grid, dim3 block, cudaStream_t st, int cluster,
                      const Args& a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MPSG_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
}

// Device scratch and launches of one solve.
struct LanczosWork {
  Context* ctx;
  int kd, grid;
  int64_t n;
  bool cluster;
  unsigned barriers = 0;
  std::shared_ptr<Buffer> buf;
  double* part;           // partial sums
  double* out;            // pinned: per step of a cycle (alpha, beta), then the norm of a combination
  unsigned* count;
  LanczosWork(Context* c, int kd_, int64_t n_) : ctx(c), kd(kd_), n(n_) {
    // one block per SM at most: co-resident, and few arrivals per barrier; short vectors are bound
    // by the FP64 pipes of the SMs that take part (22 FMAs per element at K = 5), so they spread
    grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(ctx->num_sms, (n + kVecThreads - 1) / kVecThreads));
    cluster = n <= (int64_t)kClusterBlocks * kClusterRows * kVecThreads;
    if (cluster) grid = std::min(grid, kClusterBlocks);
    const int64_t np = 3 * (int64_t)kd * grid;
    buf = alloc_buffer(ctx, np + 1);
    part = buf->ptr;
    out = ctx->h_pinned + Context::kPinnedKrylov;
    count = (unsigned*)(part + np);
    for (auto& e : ctx->krylov_ev)
      if (!e) MPSG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    MPSG_CUDA(cudaMemsetAsync(count, 0, sizeof(double), ctx->stream));
  }
  GridBarrier barrier(int n_barriers) {
    GridBarrier b{cluster ? nullptr : count, (barriers + 1) * (unsigned)grid,
                  ctx->wait_err + kWaitKrylov};
    barriers += (unsigned)n_barriers;
    return b;
  }
  template <class Args>
  void run(void (*kernel)(Args), Args& a) {
    ctx->kernel_launches++;
    if (cluster) {
      launch_clustered(kernel, dim3((unsigned)grid), dim3(kVecThreads), ctx->stream, grid, a);
      return;
    }
    void* p[] = {&a};
    MPSG_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(kVecThreads), p, 0,
                                          ctx->stream));
  }
  // Krylov step number i of the cycle: w against V[0..K), next <- the rest normalised
  void step(int i, const std::vector<DeviceTensor>& V, int K, DeviceTensor& w, DeviceTensor& next) {
    StepArgs a;
    for (int j = 0; j < K; ++j) a.V[j] = V[j].data();
    a.w = w.data();
    a.next = next.data();
    a.part = part;
    a.out = out + 2 * i;
    a.K = K;
    a.n = n;
    a.bar = barrier(3);
    run(K <= 4 ? krylov_step_kernel<4> : K <= 8 ? krylov_step_kernel<8>
        : K <= 16 ? krylov_step_kernel<16> : krylov_step_kernel<32>, a);
  }
  // x <- sum_j c_j V_j, normalised
  void combine(const std::vector<const double*>& V, const double* c, double* x) {
    CombineArgs a;
    for (size_t j = 0; j < V.size(); ++j) {
      a.V[j] = V[j];
      a.c[j] = c[j];
    }
    a.x = x;
    a.part = part;
    a.out = out + 2 * kd;
    a.K = (int)V.size();
    a.n = n;
    a.bar = barrier(1);
    run(krylov_combine_kernel, a);
  }
  void restart(std::vector<DeviceTensor>& V, const std::vector<double>& U, int K, int keep) {
    if (n == 0) return;
    RestartArgs a;
    for (int j = 0; j < K; ++j) a.V[j] = V[j].data();
    for (int i = 0; i < keep; ++i)
      for (int j = 0; j < K; ++j) a.U[i * K + j] = U[j + K * i];
    a.K = K;
    a.keep = keep;
    a.n = n;
    auto kern = K <= 8 ? krylov_restart_kernel<8> : krylov_restart_kernel<32>;
    const unsigned g = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>((n + kVecThreads - 1) / kVecThreads, (int64_t)ctx->num_sms * 4));
    kern<<<g, kVecThreads, 0, ctx->stream>>>(a);
    MPSG_CUDA(cudaGetLastError());
    ctx->kernel_launches++;
  }
  // The end of what has been queued so far, as number i, and the wait for it (at most kLag + 1 later ones may
  // have been marked by then). Kernels write their results into pinned memory, where they are after the wait.
  static constexpr int kLag = 2;
  static_assert(kLag + 1 < sizeof(Context::krylov_ev) / sizeof(cudaEvent_t), "events in flight");
  void mark(int i) { MPSG_CUDA(cudaEventRecord(ctx->krylov_ev[i & 3], ctx->stream)); }
  void wait(int i) {
    MPSG_CUDA(cudaEventSynchronize(ctx->krylov_ev[i & 3]));
    check_waits(ctx);
  }
  double alpha(int i) const { return ((volatile double*)out)[2 * i]; }
  double beta(int i) const { return ((volatile double*)out)[2 * i + 1]; }
  double norm() const { return ((volatile double*)out)[2 * kd]; }
};

}  // namespace

// The recurrence runs ahead on the device: matrix-vector products and Krylov steps are queued while the host
// looks at the coefficients of the step kLag before, so the device does not wait for it, and a start
// vector that is refused or a step whose remainder is below tol (which ends the solve at that step) is
// known at most kLag products later; what was queued after it is dropped. At the end of a cycle (krylovdim -
// kept vectors of products) the host decomposes the projected matrix (a few us for its at most 32 x 32
// elements) and decides.
EigResult eigsolve_heff2(Context* ctx, const DeviceTensor& x0, const DeviceTensor& envL,
                         const DeviceTensor& envR, const DeviceTensor& W1, const DeviceTensor& W2,
                         int krylovdim, int maxiter, double tol, int precision) {
  if (krylovdim < 2) throw Error(kErrArgument, "krylovdim must be at least 2");
  if (krylovdim > kMaxKrylov) throw Error(kErrArgument, "krylovdim must be at most 32");
  if (maxiter < 1) throw Error(kErrArgument, "maxiter must be at least 1");
  if (x0.meta.total == 0) throw Error(kErrArgument, "eigsolve: zero start vector");
  auto op = heff_create(ctx, x0.meta, envL, envR, W1, W2, precision);
  const int kd = krylovdim, keep = std::max(1, 3 * kd / 5);
  LanczosWork Wk(ctx, kd, x0.meta.total);
  std::vector<DeviceTensor> V;
  for (int j = 0; j <= kd; ++j) V.push_back(new_tensor(ctx, x0.meta, false));
  const double one = 1.0;
  Wk.combine({x0.data()}, &one, V[0].data());
  Wk.mark(3);  // (its event is not reused before step 3)
  std::vector<double> H(kd * kd, 0.0), D(kd), U(kd * kd);  // column-major, leading dimension kd
  auto at = [&](int i, int j) -> double& { return H[i + kd * j]; };
  int have = 1, numops = 0;  // basis vectors at the cycle's start (the newest not yet multiplied)
  for (int numiter = 1;; ++numiter) {
    bool more = true;
    for (int K = have; K <= kd && more; ++K) {
      const int i = K - have, before = i - LanczosWork::kLag;
      DeviceTensor w = heff_apply(*op, V[K - 1]);
      Wk.step(i, V, K, w, V[K]);
      Wk.mark(i);
      if (before >= 0) {
        Wk.wait(before);
        more = Wk.beta(before) > tol || std::isnan(Wk.beta(before));
      }
      if (numiter == 1 && i == 0) {
        MPSG_CUDA(cudaEventSynchronize(ctx->krylov_ev[3]));
        if (!(Wk.norm() > 0)) throw Error(kErrArgument, "eigsolve: zero start vector");
      }
      if (K == kd || !more) Wk.wait(i);
    }
    int K = have;
    double beta = 0.0;
    for (;; ++K) {
      at(K - 1, K - 1) += Wk.alpha(K - have);
      beta = Wk.beta(K - have);
      ++numops;
      if (K == kd || beta <= tol) break;
      at(K, K - 1) = at(K - 1, K) = beta;
    }
    std::vector<double> Hk(K * K);
    for (int j = 0; j < K; ++j)
      for (int i = 0; i < K; ++i) Hk[i + K * j] = at(i, j);
    small_eigh(K, Hk.data(), D.data(), U.data());
    const double normres = std::fabs(beta * U[K - 1]);
    const bool converged = normres <= tol;
    if (converged || beta <= tol || numiter >= maxiter) {
      std::vector<const double*> xv(K);
      for (int j = 0; j < K; ++j) xv[j] = V[j].data();
      DeviceTensor x = new_tensor(ctx, x0.meta, false);
      Wk.combine(xv, U.data(), x.data());
      EigResult R;
      R.value = D[0];
      R.vec = x;
      R.normres = normres;
      R.numiter = numiter;
      R.numops = numops;
      R.converged = converged;
      return R;
    }
    // thick restart: the lowest `keep` Ritz vectors, then the normalised remainder
    Wk.restart(V, U, K, keep);
    std::swap(V[keep], V[kd]);
    std::fill(H.begin(), H.end(), 0.0);
    for (int i = 0; i < keep; ++i) {
      at(i, i) = D[i];
      if (keep < kd) at(keep, i) = at(i, keep) = beta * U[(K - 1) + K * i];
    }
    have = keep + 1;
  }
}

}  // namespace mpsg
