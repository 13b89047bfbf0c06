// GMRES on the FP64 AIC (solve_gmres!, src/FLOWPanel_linearsolver.jl:110-157:
// Krylov.jl 0.9's gmres with memory=50, atol=rtol=sqrt(eps), restart=false),
// and GMRES-IR: restarted GMRES right-preconditioned by the FP32 LU factors,
// started from the refined iterate, for the mixed-precision form.
//
// Arnoldi uses classical Gram-Schmidt applied twice (two fused passes of
// dot products and updates per step instead of j sequential MGS steps); the
// small Hessenberg least-squares problem (Givens rotations) runs on the host.
// Stop test as Krylov.jl: the residual estimate <= atol + rtol ||r0||.
//
// A step is seven short kernels (A v is HBM-bound: 8 N^2 bytes; the others are
// latency-bound), launched programmatically dependent. Nothing of it waits for
// the host: the last kernel normalises V_{j+1} and leaves column j of the
// Hessenberg matrix in mapped host memory, and the host, which only decides
// when to stop, runs its rotations kAhead steps behind the launches. N = 3,828 (A,
// 117 MB, about fills L2): 38 us a step over 211 steps, of which A v 23 (41 over 350:
// the passes over the basis grow); with a host synchronisation and plain loads 153.
// 480 unknowns 87 -> 20 us a step, 12,000 320 -> 210.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "fp_internal.cuh"

namespace fpb {

constexpr int kDotThreads = 256;

// What these passes move is small (4 MB of basis vectors, or the matrix from L2
// and HBM), so memory latency over the bytes in flight is what they take; plain
// loads were scheduled one or two ahead of their use whatever the source said
// (A v 33 to 68 us at N = 3,828, the projections 19 to 29). So every operand is
// copied to shared memory by cp.async, all of it in flight at once, and summed
// from there, in the order of the plain loops.
//
// The step's kernels start before the previous one has ended (griddep_wait), so
// what that one writes is read only after it.
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// a[0 .. count) -> dst, count rounded up to whole 16 bytes (the vectors' leading dimension is even)
__device__ __forceinline__ void stage(double* dst, const double* a, int count) {
  for (int q = 2 * threadIdx.x; q < count; q += 2 * blockDim.x) cp16(dst + q, a + q);
}

// h[i] = V_i . w, i < nv: one CTA a vector, 4,096 rows staged at a time
constexpr int kDotRows = 4096;
__global__ void __launch_bounds__(kDotThreads)
k_dots(const double* V, int64_t ld, int nv, const double* w, int64_t n, double* h) {
  extern __shared__ __align__(16) double st[];
  __shared__ double red[kDotThreads / 32];
  griddep_wait();
  griddep_launch();
  const int i = blockIdx.x;
  double s = 0.0;
  for (int64_t r0 = 0; r0 < n; r0 += kDotRows) {
    const int m = (int)imin64(kDotRows, n - r0);
    __syncthreads();
    stage(st, V + (int64_t)i * ld + r0, m);
    stage(st + kDotRows, w + r0, m);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    for (int r = threadIdx.x; r < m; r += kDotThreads) s += st[r] * st[kDotRows + r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kDotThreads / 32; ++q) t += red[q];
    h[i] = t;
  }
}

// w -= sum_i h[i] V_i: 32 rows a CTA, 128 vectors staged at a time by 256
// threads, the rows' chains by the first warp
constexpr int kSubRows = 32, kSubVecs = 128, kSubThreads = 256;
__global__ void __launch_bounds__(kSubThreads)
k_sub_Vh(const double* V, int64_t ld, int nv, const double* h, double* w, int64_t n) {
  extern __shared__ __align__(16) double st[];   // two of [vector][row], then the coefficients
  griddep_wait();
  griddep_launch();
  const int64_t r0 = (int64_t)blockIdx.x * kSubRows, r = r0 + threadIdx.x;
  const bool mine = threadIdx.x < kSubRows && r < n;
  double* const sh = st + 2 * kSubVecs * kSubRows;
  auto issue = [&](int i0) {
    double* dst = st + ((i0 / kSubVecs) & 1) * kSubVecs * kSubRows;
    for (int e = threadIdx.x; e < min(kSubVecs, nv - i0) * (kSubRows / 2); e += kSubThreads) {
      const int i = e / (kSubRows / 2), q = 2 * (e % (kSubRows / 2));
      cp16(dst + i * kSubRows + q, V + (int64_t)(i0 + i) * ld + r0 + q);   // ld is a multiple of 64
    }
    cp_commit();
  };
  issue(0);
  double s = mine ? w[r] : 0.0;
  for (int i0 = 0; i0 < nv; i0 += kSubVecs) {
    const int m = min(kSubVecs, nv - i0);
    if (i0 + kSubVecs < nv) { issue(i0 + kSubVecs); cp_wait<1>(); } else { cp_wait<0>(); }
    if ((int)threadIdx.x < m) sh[threadIdx.x] = h[i0 + threadIdx.x];
    __syncthreads();
    const double* v = st + ((i0 / kSubVecs) & 1) * kSubVecs * kSubRows + threadIdx.x;
    if (mine)
#pragma unroll 8
      for (int i = 0; i < m; ++i) s -= sh[i] * v[i * kSubRows];
    __syncthreads();
  }
  if (mine) w[r] = s;
}

// parts of w = A v: 128 rows and one of kGemvSplitHost column ranges a CTA, 16
// columns a stage; the first stages of A are under way before v is there
// Three stages, four CTAs an SM. A step at 2,000, 3,828, 6,300, 8,000 and 12,000 unknowns
// takes 23.5, 38.0, 81, 105 and 210 us; with two stages 23.8, 39.2, 71, 117 and 203, with
// four (three CTAs) 23.8, 48.9, 80, 127 and 235.
constexpr int kMvRows = 128, kMvCols = 16, kMvStages = 3;
constexpr size_t kMvSmem = (size_t)kMvStages * kMvCols * (kMvRows + 1) * sizeof(double);
__global__ void __launch_bounds__(kMvRows)
k_matvec(const double* __restrict__ A, int64_t lda, int64_t n, const double* v, double* part) {
  extern __shared__ __align__(16) double st[];
  double* const sv = st + kMvStages * kMvCols * kMvRows;   // v of each stage's columns
  const int64_t i0 = (int64_t)blockIdx.x * kMvRows, i = i0 + threadIdx.x;
  const int64_t cs = (n + gridDim.y - 1) / gridDim.y;
  const int64_t c0 = blockIdx.y * cs, c1 = imin64(n, c0 + cs);
  const int steps = c1 > c0 ? (int)((c1 - c0 + kMvCols - 1) / kMvCols) : 0;
  const int rows = (int)imin64(kMvRows, lda - i0);
  auto issue = [&](int t) {
    if (t < steps) {
      const int64_t j0 = c0 + (int64_t)t * kMvCols;
      double* dst = st + (t % kMvStages) * kMvCols * kMvRows;
#pragma unroll
      for (int u = 0; u < kMvCols / 2; ++u) {   // 64 threads a column
        const int e = threadIdx.x + u * kMvRows, c = e / (kMvRows / 2), q = 2 * (e % (kMvRows / 2));
        if (j0 + c < c1 && q < rows) cp16(dst + c * kMvRows + q, A + (j0 + c) * lda + i0 + q);
      }
    }
    cp_commit();
  };
#pragma unroll
  for (int t = 0; t < kMvStages - 1; ++t) issue(t);
  griddep_wait();
  griddep_launch();
  double s = 0.0;
  for (int t = 0; t < steps; ++t) {
    const int64_t j0 = c0 + (int64_t)t * kMvCols;
    const int m = (int)imin64(kMvCols, c1 - j0);
    double* const svt = sv + (t % kMvStages) * kMvCols;
    if ((int)threadIdx.x < m) svt[threadIdx.x] = v[j0 + threadIdx.x];
    cp_wait<kMvStages - 2>();
    __syncthreads();   // stage t has landed; the one before it is read
    issue(t + kMvStages - 1);
    const double* a = st + (t % kMvStages) * kMvCols * kMvRows + threadIdx.x;
    if (m == kMvCols) {
#pragma unroll
      for (int c = 0; c < kMvCols; ++c) s += a[c * kMvRows] * svt[c];
    } else {
      for (int c = 0; c < m; ++c) s += a[c * kMvRows] * svt[c];
    }
  }
  cp_wait<0>();
  if (i < n) part[blockIdx.y * n + i] = s;
}
__global__ void k_matvec_sum(const double* part, int64_t n, double* w) {
  griddep_wait();
  griddep_launch();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
#pragma unroll
  for (int p = 0; p < kGemvSplitHost; ++p) s += part[p * n + i];
  w[i] = s;
}

// v_next = w / ||w|| (every CTA forms the norm), and to the host column j of the
// Hessenberg matrix: h + h2, then ||w||
__global__ void __launch_bounds__(kDotThreads)
k_next(const double* w, int64_t n, double* v_next, const double* h, const double* h2, int nv, double* out) {
  extern __shared__ __align__(16) double st[];
  __shared__ double red[kDotThreads / 32];
  griddep_wait();
  griddep_launch();
  double s = 0.0;
  for (int64_t r0 = 0; r0 < n; r0 += kDotRows) {
    const int m = (int)imin64(kDotRows, n - r0);
    __syncthreads();
    stage(st, w + r0, m);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    for (int r = threadIdx.x; r < m; r += kDotThreads) s += st[r] * st[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  for (int q = 0; q < kDotThreads / 32; ++q) t += red[q];
  const double norm = sqrt(t), alpha = 1.0 / norm;
  const int64_t r = (int64_t)blockIdx.x * kDotThreads + threadIdx.x;
  if (r < n) v_next[r] = alpha * w[r];
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < nv; i += kDotThreads) out[i] = h[i] + h2[i];
    if (threadIdx.x == 0) out[nv] = norm;
  }
}

// u = V y (nv columns)
__global__ void k_Vy(const double* __restrict__ V, int64_t ld, int nv, const double* __restrict__ y,
                     double* __restrict__ u, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  double s = 0.0;
  for (int i = 0; i < nv; ++i) s += y[i] * V[(int64_t)i * ld + r];
  u[r] = s;
}

__global__ void k_scale(const double* __restrict__ a, double alpha, double* __restrict__ b, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) b[r] = alpha * a[r];
}

__global__ void k_add(double* __restrict__ x, const double* __restrict__ u, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) x[r] += u[r];
}

__global__ void k_to_f32(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) b[r] = (float)a[r];
}
__global__ void k_to_f64(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) b[r] = (double)a[r];
}

int colnorm2(fp_ctx* c, const double* a, int64_t n, int64_t lda, int64_t k, double* d_out);

namespace {
struct Gm {
  fp_ctx* c;
  int64_t n, ld;
  unsigned g1;
  int norm2(const double* a, double* out) {
    if (int rc = colnorm2(c, a, n, ld, 1, c->d_h)) return rc;
    FP_CUDA_TRY(c->err, cudaMemcpyAsync(out, c->d_h, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    FP_CUDA_TRY(c->err, cudaStreamSynchronize(c->stream));
    return FP_OK;
  }
  // u <- M^-1 u with the context's factors (FP64 in place, or the FP32 ones)
  int precond(double* u) {
    if (c->factored == FP_PREC_FP64) return lu_solve<double>(c, c->d_LU, n, ld, c->d_ipiv, u, ld, 1, false);
    k_to_f32<<<g1, 256, 0, c->stream>>>(u, c->d_w32, n);
    ++c->nlaunch;
    if (int rc = lu_solve<float>(c, c->d_G32, n, ld, c->d_ipiv, c->d_w32, ld, 1, false)) return rc;
    k_to_f64<<<g1, 256, 0, c->stream>>>(c->d_w32, u, n);
    ++c->nlaunch;
    FP_CUDA_TRY(c->err, cudaGetLastError());
    return FP_OK;
  }
};

// Device buffers for a basis of `cap` vectors: d_V holds the work vector w,
// the correction u, then V_0 .. V_cap (cap + 3 columns of ld); d_h holds the
// norms, two projection vectors of cap + 1 entries and y; h_gm (mapped host
// memory) the Hessenberg columns of kRing steps, cap + 2 entries each. `keep`
// columns of the old basis (w and u included) and the columns the host has not
// read yet are carried over when it grows.
constexpr int kAhead = 2, kRing = kAhead + 1;
int ensure_basis(fp_ctx* c, int cap, int keep) {
  if (c->cap_gmres_m >= cap) return FP_OK;
  const int64_t ld = c->ld;
  for (cudaEvent_t& ev : c->ev_gm)
    if (!ev) FP_CUDA_TRY(c->err, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  double* V = nullptr;
  double* h = nullptr;
  double* ring = nullptr;
  // the basis first: if there is no room for it, no host memory is pinned
  cudaError_t e = cudaMalloc(&V, (size_t)(cap + 3) * ld * sizeof(double));
  if (!e) e = cudaMalloc(&h, (size_t)(3 * ((size_t)cap + 1) + 16) * sizeof(double));
  if (!e) e = cudaHostAlloc(&ring, (size_t)kRing * ((size_t)cap + 2) * sizeof(double), cudaHostAllocMapped);
  if (!e && c->d_V && keep > 0)
    e = cudaMemcpyAsync(V, c->d_V, (size_t)keep * ld * sizeof(double), cudaMemcpyDeviceToDevice, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  if (e) {
    cudaFree(V);
    cudaFree(h);
    if (ring) cudaFreeHost(ring);
    cudaGetLastError();
    return c->err.set(FP_ECUDA, std::string("GMRES basis: ") + cudaGetErrorString(e));
  }
  if (c->d_V) cudaFree(c->d_V);
  if (c->d_h) cudaFree(c->d_h);
  if (c->h_gm) {
    const size_t old = (size_t)c->cap_gmres_m + 2;
    for (int q = 0; q < kRing; ++q) std::memcpy(ring + q * (size_t)(cap + 2), c->h_gm + q * old, old * sizeof(double));
    cudaFreeHost(c->h_gm);
  }
  c->h_gm = ring;
  c->d_V = V;
  c->d_h = h;
  c->cap_gmres_m = cap;
  return FP_OK;
}
}  // namespace

// GMRES for k right-hand sides, one after the other (as gmres(A, b::AbstractMatrix)
// does, src/FLOWPanel_linearsolver.jl:151-157), each from x = 0 unless
// `precondition` (GMRES-IR: from the refined iterate, right-preconditioned by
// the context's LU factors: the FP32 ones, or FP64 factors whose block-local
// pivots are not certified).
//  * Default (the reference's Krylov.jl 0.9 gmres with restart = false): one
//    Arnoldi process whose basis grows past `memory` (a storage hint) until
//    the Givens estimate of the residual norm falls to atol + rtol ||r0|| or
//    itmax steps (2N) are taken; a breakdown (h_{j+1,j} <= eps^(3/4)) ends it.
//  * gmres_restart != 0, and GMRES-IR: GMRES(memory), restarted from the true
//    residual, which must itself meet the tolerance.
int gmres_solve(fp_ctx* c, const double* b, double* x, int64_t k, const fp_solve_opts& o,
                bool precondition, int* iters, double* relres) {
  const int64_t n = c->N, ld = c->ld;
  const int mem = o.gmres_memory > 0 ? o.gmres_memory : 50;
  const bool restart = precondition || o.gmres_restart != 0;
  const double eps = 2.220446049250313e-16;
  const double btol = std::pow(eps, 0.75);
  const double atol = o.gmres_atol >= 0 ? o.gmres_atol : std::sqrt(eps);
  const double rtol = o.gmres_rtol >= 0 ? o.gmres_rtol : std::sqrt(eps);
  const int64_t itmax = o.gmres_itmax > 0 ? o.gmres_itmax : 2 * n;
  if (precondition && c->factored != FP_PREC_MIXED && c->factored != FP_PREC_FP64)
    return c->err.set(FP_ESTATE, "GMRES-IR needs LU factors");
  if (int rc = ensure_basis(c, (int)std::min<int64_t>(mem, itmax), 0)) return rc;
  if (!c->d_part) FP_CUDA_TRY(c->err, cudaMalloc(&c->d_part, (size_t)kGemvSplitHost * 4 * c->capN * sizeof(double)));
  Gm G{c, n, ld, (unsigned)((n + 255) / 256)};
  int total = 0;
  double worst = 0.0;
  bool all_conv = true;
  // host side of the Arnoldi process: column j of the rotated Hessenberg
  // matrix (j + 2 entries), the rotations and the rotated right-hand side
  std::vector<std::vector<double>> H;
  std::vector<double> cs, sn, g, y;
  for (int64_t q = 0; q < k; ++q) {
    const double* bq = b + q * ld;
    double* xq = x + q * ld;
    if (!precondition) FP_CUDA_TRY(c->err, cudaMemsetAsync(xq, 0, n * sizeof(double), c->stream));
    double bn2 = 0;
    if (int rc = G.norm2(bq, &bn2)) return rc;
    const double bnorm = std::sqrt(bn2);
    // Krylov.jl: eps = atol + rtol ||r0||, with r0 = b from x = 0; GMRES-IR
    // measures against ||b|| too
    const double target = atol + rtol * bnorm;
    // r = b - A x in w
    if (int rc = gemv_residual(c, c->d_G, n, ld, xq, bq, c->d_V, 1)) return rc;
    double beta2 = 0;
    if (int rc = G.norm2(c->d_V, &beta2)) return rc;
    double beta = std::sqrt(beta2);
    int it = 0;
    bool conv = beta <= target;
    while (!conv && it < itmax) {
      k_scale<<<G.g1, 256, 0, c->stream>>>(c->d_V, 1.0 / beta, c->d_V + 2 * ld, n);
      ++c->nlaunch;
      H.clear(); cs.clear(); sn.clear();
      g.assign(1, beta);
      int kd = 0;
      bool solved = false;
      // launches of step j: w = A V_j (or A M^-1 V_j), orthogonalised twice,
      // V_{j+1}, column j of the Hessenberg matrix to its slot of the ring
      auto launch = [&](int j) -> int {
        if (j + 1 > c->cap_gmres_m) {   // the basis outgrows its storage hint: room for V_{j+1}
          const int cap2 = (int)std::min<int64_t>(2 * (int64_t)c->cap_gmres_m, itmax);
          if (int rc = ensure_basis(c, std::max(cap2, j + 1), j + 3)) return rc;
        }
        double* const w = c->d_V;
        double* const V = c->d_V + 2 * ld;
        double* const dh = c->d_h + 8;
        double* const dh2 = dh + c->cap_gmres_m + 1;
        const double* src = V + (size_t)j * ld;
        if (precondition) {
          double* const u = c->d_V + ld;
          FP_CUDA_TRY(c->err, cudaMemcpyAsync(u, src, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
          if (int rc = G.precond(u)) return rc;
          src = u;
        }
        const dim3 gm((unsigned)((n + kMvRows - 1) / kMvRows), kGemvSplitHost);
        const unsigned gs = (unsigned)((n + kSubRows - 1) / kSubRows);
        constexpr size_t sm_dot = 2 * kDotRows * sizeof(double), sm_next = kDotRows * sizeof(double),
                         sm_sub = (size_t)(2 * kSubRows + 1) * kSubVecs * sizeof(double);
        static SmemAttr am, ad, as;
        FP_CUDA_TRY(c->err, am.ensure(k_matvec, (int)kMvSmem));
        FP_CUDA_TRY(c->err, ad.ensure(k_dots, (int)sm_dot));
        FP_CUDA_TRY(c->err, as.ensure(k_sub_Vh, (int)sm_sub));
        launch_k(true, k_matvec, gm, dim3(kMvRows), kMvSmem, c->stream, c->d_G, ld, n, src, c->d_part);
        launch_k(true, k_matvec_sum, dim3(G.g1), dim3(256), 0, c->stream, c->d_part, n, w);
        for (double* hq : {dh, dh2}) {   // classical Gram-Schmidt, twice
          launch_k(true, k_dots, dim3(j + 1), dim3(kDotThreads), sm_dot, c->stream, V, ld, j + 1, w, n, hq);
          launch_k(true, k_sub_Vh, dim3(gs), dim3(kSubThreads), sm_sub, c->stream, V, ld, j + 1, hq, w, n);
        }
        launch_k(true, k_next, dim3(G.g1), dim3(kDotThreads), sm_next, c->stream, w, n, V + (size_t)(j + 1) * ld, dh, dh2,
                 j + 1, c->h_gm + (size_t)(j % kRing) * (c->cap_gmres_m + 2));
        c->nlaunch += 7;
        FP_CUDA_TRY(c->err, cudaGetLastError());
        FP_CUDA_TRY(c->err, cudaEventRecord(c->ev_gm[j % kRing], c->stream));
        return FP_OK;
      };
      // a preconditioned step is a whole solve: none is launched in vain
      const int ahead = precondition ? 0 : kAhead;
      const int64_t steps = std::min<int64_t>(restart ? mem : itmax, itmax - it);
      int queued = 0;
      for (int j = 0; j < steps; ++j) {
        // ahead only in the basis there is: it grows for a step that is taken
        for (; queued < steps && (queued == j || (queued <= j + ahead && queued + 1 <= c->cap_gmres_m)); ++queued)
          if (int rc = launch(queued)) return rc;
        FP_CUDA_TRY(c->err, cudaEventSynchronize(c->ev_gm[j % kRing]));
        const double* hj = c->h_gm + (size_t)(j % kRing) * (c->cap_gmres_m + 2);
        const double hn = hj[j + 1];
        H.emplace_back(j + 2);
        std::vector<double>& Hj = H.back();
        for (int i = 0; i <= j; ++i) Hj[i] = hj[i];
        Hj[j + 1] = hn;
        const bool breakdown = hn <= btol;
        // Givens rotations
        for (int i = 0; i < j; ++i) {
          const double t = cs[i] * Hj[i] + sn[i] * Hj[i + 1];
          Hj[i + 1] = -sn[i] * Hj[i] + cs[i] * Hj[i + 1];
          Hj[i] = t;
        }
        const double den = std::hypot(Hj[j], Hj[j + 1]);
        cs.push_back(den > 0 ? Hj[j] / den : 1.0);
        sn.push_back(den > 0 ? Hj[j + 1] / den : 0.0);
        Hj[j] = den;
        Hj[j + 1] = 0.0;
        g.push_back(-sn[j] * g[j]);
        g[j] = cs[j] * g[j];
        ++it;
        kd = j + 1;
        solved = std::fabs(g[j + 1]) <= target;
        if (solved || breakdown) break;
      }
      // y = R^-1 g (upper triangular kd x kd), x += V y (preconditioned)
      y.assign(kd, 0.0);
      for (int i = kd - 1; i >= 0; --i) {
        double s = g[i];
        for (int l = i + 1; l < kd; ++l) s -= H[l][i] * y[l];
        y[i] = s / H[i][i];
      }
      double* const w = c->d_V;
      double* const u = c->d_V + ld;
      double* const V = c->d_V + 2 * ld;
      double* const dh = c->d_h + 8;
      FP_CUDA_TRY(c->err, cudaMemcpyAsync(dh, y.data(), kd * sizeof(double), cudaMemcpyHostToDevice, c->stream));
      k_Vy<<<G.g1, 256, 0, c->stream>>>(V, ld, kd, dh, u, n);
      ++c->nlaunch;
      if (precondition)
        if (int rc = G.precond(u)) return rc;
      k_add<<<G.g1, 256, 0, c->stream>>>(xq, u, n);
      ++c->nlaunch;
      FP_CUDA_TRY(c->err, cudaGetLastError());
      if (int rc = gemv_residual(c, c->d_G, n, ld, xq, bq, w, 1)) return rc;
      if (int rc = G.norm2(w, &beta2)) return rc;
      beta = std::sqrt(beta2);
      // restarted: the true residual decides; one Arnoldi process: its estimate
      conv = restart ? beta <= target : solved;
      if (!restart) break;
    }
    total += it;
    worst = std::max(worst, bnorm > 0 ? beta / bnorm : beta);
    all_conv = all_conv && conv;
  }
  *iters = total;
  *relres = worst;
  if (!all_conv) return c->err.set(FP_ENOCONV, "GMRES did not reach its tolerance");
  return FP_OK;
}

}  // namespace fpb
