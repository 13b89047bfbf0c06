// Several right-hand sides at once: the sweeps with the LU factors (k_trsm) and
// the FP64 residual (k_resid).
//
// A sweep is a chain of n / 128 dependent blocks, so what counts is the time from
// one block's solution to the next one's, and how few sweeps there are: up to
// 32 right-hand sides share one. Refining 21 of them at n = 12,000 in the mixed
// form (five times two sweeps and a residual) took 31.1 ms in groups of 8, 4 and 1
// with 64-row blocks and residuals of 4 a pass, and takes 7.4 ms; the FP64
// sweeps of 21 fell from 7.4 to 2.5 ms.
#include "fp_internal.cuh"

namespace fpb {
namespace ts {

constexpr int SB = 128, NT = 256;
constexpr int kSpin = 1 << 22;
// columns of a staged chunk of a 128-row tile: 64 KB
template <class T> __host__ __device__ constexpr int chunk() { return sizeof(T) == 4 ? 128 : 64; }
// pitch of a row of KR right-hand sides: whole 16-byte loads, few bank conflicts down a column
template <class T, int KR> __host__ __device__ constexpr int ypitch() { return KR + 16 / (int)sizeof(T); }
template <class T, int KR> constexpr size_t smem() {
  return (size_t)2 * chunk<T>() * SB * sizeof(T) + (size_t)SB * ypitch<T, KR>() * sizeof(T);
}

__device__ __forceinline__ void cp16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// acc[2 rows][KQ] += tile (KC columns of 128 rows, [column][row]) times Y ([column][right-hand side])
template <class T, int KQ, int YP>
__device__ __forceinline__ void product(const T* __restrict__ tile, const T* __restrict__ Y, int cols, T (&acc)[2][KQ]) {
  struct alignas(2 * sizeof(T)) Two { T a, b; };
#pragma unroll 4
  for (int l = 0; l < cols; ++l) {
    const Two a = *reinterpret_cast<const Two*>(tile + (size_t)l * SB);
    T y[KQ];
#pragma unroll
    for (int q = 0; q < KQ; q += 2) {   // KQ is even
      const Two v = *reinterpret_cast<const Two*>(Y + (size_t)l * YP + q);
      y[q] = v.a;
      y[q + 1] = v.b;
    }
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      acc[0][q] += a.a * y[q];
      acc[1][q] += a.b * y[q];
    }
  }
}

// One sweep over all blocks for kr <= KR right-hand sides (B: column q at q ldb).
// CTAs take blocks by ticket, in sweep order, so a CTA waits only for blocks of
// CTAs already running. Block b: for every earlier block but the predecessor,
// as it is published, acc -= T(b, s) x_s; x' = inv(D_b) acc; then
// x_b = x' - M_b x_p with M_b = inv(D_b) T(b, p) (k_mprev), so that the step of the
// chain is one product. The tiles stream through two 64 KB buffers, always
// one chunk ahead, whatever is waited for. Warp w: rows 64 (w / 4) + 2 lane,
// right-hand sides KR / 4 (w % 4)..: a column of the product reads 32 words of
// shared memory per bank for 24 cycles of FMAs a scheduler.
template <class T, bool LOWER, int KR>
__global__ void __launch_bounds__(NT, 1)
k_trsm(const T* __restrict__ A, int64_t lda, int64_t n, const T* __restrict__ Dinv128, const T* __restrict__ Mprev,
       T* B, int64_t ldb, int kr, unsigned* flags, unsigned* ticket, int* __restrict__ status) {
  constexpr int KC = chunk<T>(), NC = SB / KC, KQ = KR / 4, YP = ypitch<T, KR>(), V = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char sm[];
  T* const buf = reinterpret_cast<T*>(sm);
  T* const Y = buf + (size_t)2 * KC * SB;
  __shared__ int blk, stop;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = 64 * (warp >> 2) + 2 * lane, q0 = KQ * (warp & 3);
  const int64_t nblk = (n + SB - 1) / SB;
  for (;;) {
    __syncthreads();
    if (tid == 0) { blk = (int)atomicAdd(ticket, 1u); stop = 0; }
    __syncthreads();
    const int64_t tk = blk;
    if (tk >= nblk) return;
    const int64_t b = LOWER ? tk : nblk - 1 - tk, k0 = b * SB;
    const int nb = (int)imin64(SB, n - k0);
    const T* const Di = Dinv128 + (b * 2 + (LOWER ? 0 : 1)) * SB * SB;
    const T* const Mp = Mprev + (b * 2 + (LOWER ? 0 : 1)) * SB * SB;
    auto block_at = [&](int64_t s) { return LOWER ? s : nblk - 1 - s; };
    const int64_t nt = tk > 0 ? tk - 1 : 0;   // tiles before the predecessor's
    const int64_t total = (nt + 1 + (tk > 0 ? 1 : 0)) * NC;
    // chunk i of the tile sequence T(b, 0) .. , inv(D_b), M_b into buffer i & 1
    auto issue = [&](int64_t i) {
      if (i < total) {
        const int64_t s = i / NC;
        const int kk = (int)(i % NC) * KC;
        T* dst = buf + (size_t)(i & 1) * KC * SB;
        const T* src;
        int64_t ld = SB;
        int rows = SB, cols = KC;
        if (s < nt) {
          const int64_t c0 = block_at(s) * SB;
          src = A + (c0 + kk) * lda + k0;
          ld = lda;
          rows = nb;
          cols = (int)imin64(KC, n - c0 - kk);
        } else {
          src = (s == nt ? Di : Mp) + (size_t)kk * SB;
        }
        for (int e = tid; e < KC * (SB / V); e += NT) {
          const int l = e / (SB / V), r = (e % (SB / V)) * V;
          const int bytes = l < cols ? max(0, min(V, rows - r)) * (int)sizeof(T) : 0;
          cp16(dst + (size_t)l * SB + r, bytes ? src + (size_t)l * ld + r : src, bytes);
        }
      }
      cp_commit();
    };
    // block s's solution to Y once it is published (bounded)
    auto fetch = [&](int64_t s) -> bool {
      const int64_t cb = block_at(s), c0 = cb * SB;
      if (tid == 0) {
        int i = 0;
        while (load_acquire(&flags[cb]) == 0u && ++i < kSpin) {}
        if (i >= kSpin) { stop = 1; atomicOr(status, (int)DEV_TIMEOUT); }
      }
      __syncthreads();
      if (stop) return false;
      const int l = tid & (SB - 1);
#pragma unroll
      for (int q = tid / SB; q < KR; q += NT / SB) Y[l * YP + q] = q < kr && c0 + l < n ? __ldcg(&B[q * ldb + c0 + l]) : T(0);
      return true;
    };
    issue(0);
    T acc[2][KQ], x[2][KQ];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        acc[e][q] = row + e < nb && q0 + q < kr ? B[(q0 + q) * ldb + k0 + row + e] : T(0);
        x[e][q] = T(0);
      }
    for (int64_t i = 0; i < total; ++i) {
      const int64_t s = i / NC;
      const int kk = (int)(i % NC) * KC;
      issue(i + 1);
      if (kk == 0) {   // (the barrier at the end of the last chunk freed Y)
        if (s != nt) {
          if (!fetch(s < nt ? s : tk - 1)) { cp_wait<0>(); return; }
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int q = 0; q < KQ; ++q) Y[(row + e) * YP + q0 + q] = acc[e][q];
        }
      }
      cp_wait<1>();
      __syncthreads();
      T d[2][KQ];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int q = 0; q < KQ; ++q) d[e][q] = T(0);
      product<T, KQ, YP>(buf + (size_t)(i & 1) * KC * SB + row, Y + (size_t)kk * YP + q0, KC, d);
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int q = 0; q < KQ; ++q) {
          if (s < nt) acc[e][q] -= d[e][q];
          else if (s == nt) x[e][q] += d[e][q];
          else x[e][q] -= d[e][q];
        }
      __syncthreads();   // the buffer and Y are read
    }
    cp_wait<0>();
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int q = 0; q < KQ; ++q)
        if (row + e < nb && q0 + q < kr) B[(q0 + q) * ldb + k0 + row + e] = x[e][q];
    __threadfence();
    __syncthreads();
    if (tid == 0) store_release(&flags[b], 1u);
  }
}

template <class T, int KR>
static int sweeps(fp_ctx* c, const T* LU, int64_t n, int64_t lda, const T* D128, const T* Mp, T* B, int64_t ldb, int kr) {
  static SmemAttr lo, up;
  FP_CUDA_TRY(c->err, lo.ensure(k_trsm<T, true, KR>, (int)smem<T, KR>()));
  FP_CUDA_TRY(c->err, up.ensure(k_trsm<T, false, KR>, (int)smem<T, KR>()));
  const int64_t nblk = (n + SB - 1) / SB;
  const unsigned grid = (unsigned)std::min<int64_t>(nblk, num_sms());
  FP_CUDA_TRY(c->err, cudaMemsetAsync(c->d_flags, 0, (nblk + 1) * sizeof(unsigned), c->stream));
  k_trsm<T, true, KR><<<grid, NT, smem<T, KR>(), c->stream>>>(LU, lda, n, D128, Mp, B, ldb, kr, c->d_flags,
                                                              c->d_flags + nblk, c->d_status);
  FP_CUDA_TRY(c->err, cudaMemsetAsync(c->d_flags, 0, (nblk + 1) * sizeof(unsigned), c->stream));
  k_trsm<T, false, KR><<<grid, NT, smem<T, KR>(), c->stream>>>(LU, lda, n, D128, Mp, B, ldb, kr, c->d_flags,
                                                               c->d_flags + nblk, c->d_status);
  c->nlaunch += 2;
  FP_CUDA_TRY(c->err, cudaGetLastError());
  return FP_OK;
}

// ---------------------------------------------------------------------------
// r = b - A x for up to KR right-hand sides in one pass over A: 256 rows (two a
// thread) and one of kSplit column ranges a CTA, 8 columns of A and of x staged at a
// time by cp.async. With KR = 24 the FP64 pipe (2 n^2 KR) and HBM (8 n^2) take about
// the same time.
constexpr int kResRows = 256, kResThreads = 128, kResCols = 8, kResStages = 3, kSplit = 16;
template <int KR> constexpr size_t res_smem() { return (size_t)kResStages * kResCols * (kResRows + KR) * sizeof(double); }

template <int KR>
__global__ void __launch_bounds__(kResThreads)
k_resid(const double* __restrict__ A, int64_t lda, int64_t n, const double* __restrict__ xt, double* __restrict__ part) {
  extern __shared__ __align__(16) double rs[];
  const int tid = threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.x * kResRows, row = i0 + 2 * tid;
  const int64_t cs = (n + kSplit - 1) / kSplit, c0 = blockIdx.y * cs, c1 = imin64(n, c0 + cs);
  const int steps = c1 > c0 ? (int)((c1 - c0 + kResCols - 1) / kResCols) : 0;
  const int rows = (int)imin64(kResRows, lda - i0);   // lda is a multiple of 64
  auto issue = [&](int t) {
    if (t < steps) {
      const int64_t j0 = c0 + (int64_t)t * kResCols;
      double* a = rs + (size_t)(t % kResStages) * kResCols * (kResRows + KR);
      double* x = a + kResCols * kResRows;
#pragma unroll
      for (int c = 0; c < kResCols; ++c) {
        const int bytes = j0 + c < c1 && 2 * tid < rows ? 16 : 0;
        cp16(a + c * kResRows + 2 * tid, bytes ? A + (j0 + c) * lda + row : A, bytes);
      }
      for (int e = tid; e < kResCols * KR / 2; e += kResThreads) {
        const int c = e / (KR / 2), q = 2 * (e % (KR / 2));
        const int bytes = j0 + c < c1 ? 16 : 0;
        cp16(x + c * KR + q, bytes ? xt + (j0 + c) * KR + q : xt, bytes);
      }
    }
    cp_commit();
  };
  double s[2][KR];
#pragma unroll
  for (int q = 0; q < KR; ++q) s[0][q] = s[1][q] = 0.0;
#pragma unroll
  for (int t = 0; t < kResStages - 1; ++t) issue(t);
  for (int t = 0; t < steps; ++t) {
    cp_wait<kResStages - 2>();
    __syncthreads();   // stage t has landed; the one before it is read
    issue(t + kResStages - 1);
    const double* a = rs + (size_t)(t % kResStages) * kResCols * (kResRows + KR);
    const double* x = a + kResCols * kResRows;
#pragma unroll
    for (int c = 0; c < kResCols; ++c) {
      const double2 v = *reinterpret_cast<const double2*>(a + c * kResRows + 2 * tid);
#pragma unroll
      for (int q = 0; q < KR; q += 2) {
        const double2 y = *reinterpret_cast<const double2*>(x + c * KR + q);
        s[0][q] += v.x * y.x;
        s[0][q + 1] += v.x * y.y;
        s[1][q] += v.y * y.x;
        s[1][q + 1] += v.y * y.y;
      }
    }
  }
  cp_wait<0>();
  if (row < n) {
#pragma unroll
    for (int q = 0; q < KR; ++q) {
      double* p = part + ((int64_t)blockIdx.y * KR + q) * lda + row;   // lda even: whole pairs
      *reinterpret_cast<double2*>(p) = make_double2(s[0][q], s[1][q]);
    }
  }
}
// x (column q at q ld) -> xt[j][KR], zero past kr
template <int KR>
__global__ void k_xt(const double* __restrict__ x, int64_t ld, int64_t n, int kr, double* __restrict__ xt) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * KR) return;
  const int64_t j = e / KR;
  const int q = (int)(e % KR);
  xt[e] = q < kr ? x[q * ld + j] : 0.0;
}
__global__ void k_resid_sum(const double* __restrict__ part, int KR, int64_t lda, int64_t n, const double* __restrict__ b,
                            double* __restrict__ r) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int q = blockIdx.y;
  double s = 0.0;
#pragma unroll
  for (int p = 0; p < kSplit; ++p) s += part[((int64_t)p * KR + q) * lda + i];
  r[q * lda + i] = b[q * lda + i] - s;
}

template <int KR>
static int resid(fp_ctx* c, const double* A, int64_t n, int64_t lda, const double* x, const double* b, double* r, int kr) {
  const size_t need = (size_t)(kSplit + 1) * KR * lda;
  if (c->cap_res < need) {
    if (c->d_res) cudaFree(c->d_res);
    c->d_res = nullptr;
    c->cap_res = 0;
    FP_CUDA_TRY(c->err, cudaMalloc(&c->d_res, need * sizeof(double)));
    c->cap_res = need;
  }
  double* xt = c->d_res + (size_t)kSplit * KR * lda;
  static SmemAttr attr;
  FP_CUDA_TRY(c->err, attr.ensure(k_resid<KR>, (int)res_smem<KR>()));
  k_xt<KR><<<(unsigned)((n * KR + 255) / 256), 256, 0, c->stream>>>(x, lda, n, kr, xt);
  k_resid<KR><<<dim3((unsigned)((n + kResRows - 1) / kResRows), kSplit), kResThreads, res_smem<KR>(), c->stream>>>(
      A, lda, n, xt, c->d_res);
  k_resid_sum<<<dim3((unsigned)((n + 255) / 256), (unsigned)kr), 256, 0, c->stream>>>(c->d_res, KR, lda, n, b, r);
  c->nlaunch += 3;
  FP_CUDA_TRY(c->err, cudaGetLastError());
  return FP_OK;
}

}  // namespace ts

// B <- U^-1 L^-1 B for k >= 3 right-hand sides
template <class T>
int trsm_sweeps(fp_ctx* c, const T* LU, int64_t n, int64_t lda, const T* D128, const T* Mp, T* B, int64_t ldb, int64_t k) {
  for (int64_t q = 0; q < k;) {
    const int kr = (int)std::min<int64_t>(k - q, 32);
    T* b = B + q * ldb;
    int rc;
    if (kr <= 8) rc = ts::sweeps<T, 8>(c, LU, n, lda, D128, Mp, b, ldb, kr);
    else if (kr <= 16) rc = ts::sweeps<T, 16>(c, LU, n, lda, D128, Mp, b, ldb, kr);
    else if (kr <= 24) rc = ts::sweeps<T, 24>(c, LU, n, lda, D128, Mp, b, ldb, kr);
    else rc = ts::sweeps<T, 32>(c, LU, n, lda, D128, Mp, b, ldb, kr);
    if (rc) return rc;
    q += kr;
  }
  return FP_OK;
}
template int trsm_sweeps<float>(fp_ctx*, const float*, int64_t, int64_t, const float*, const float*, float*, int64_t, int64_t);
template int trsm_sweeps<double>(fp_ctx*, const double*, int64_t, int64_t, const double*, const double*, double*, int64_t,
                                 int64_t);

// r = b - A x for k >= 5 right-hand sides (leading dimension lda throughout)
int resid_multi(fp_ctx* c, const double* A, int64_t n, int64_t lda, const double* x, const double* b, double* r, int64_t k) {
  for (int64_t q = 0; q < k;) {
    const int kr = (int)std::min<int64_t>(k - q, 24);
    const int64_t o = q * lda;
    int rc;
    if (kr <= 8) rc = ts::resid<8>(c, A, n, lda, x + o, b + o, r + o, kr);
    else if (kr <= 16) rc = ts::resid<16>(c, A, n, lda, x + o, b + o, r + o, kr);
    else rc = ts::resid<24>(c, A, n, lda, x + o, b + o, r + o, kr);
    if (rc) return rc;
    q += kr;
  }
  return FP_OK;
}

}  // namespace fpb
