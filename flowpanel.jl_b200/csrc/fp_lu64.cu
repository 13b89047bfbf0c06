// FP64 LU of the FP64 form: 256-column panels in 64-column blocks, partial
// pivoting inside each 64 x 64 diagonal block (the certificate max|L21| <= 1
// says that every pivot is the one LAPACK's dgetrf picks; see fp_lu.cu).
//
// Per panel: k_panel64 factors its columns in one launch; k_strip64 swaps the
// panel's rows and forms U12 in the columns beside it; the trailing update
// follows on the FP64 tensor path (fp_lu.cu), the next panel's columns first.
//
// The panel is a chain of 256 dependent pivot steps, so its kernels are built
// for latency: one CTA of 16 warps holds 64 rows of the panel in shared memory
// for the whole panel, and blocks hand each other their factors through L2. One
// launch per 64 columns, with the rows reloaded each time and SIMT products,
// took 490 us a panel (strip and next-panel update included) where k_panel64 takes
// 141 and k_strip64 28 and 35 (captured, 3,500 rows); factorisation of 480 unknowns
// 0.95 -> 0.49 ms, 1,840 3.47 -> 1.65, 6,300 16.7 -> 9.5, 12,000 58.9 -> 49.1.
#include "fp_internal.cuh"

namespace fpb {
namespace p64 {

constexpr int R = 64;                // rows of a CTA, columns of a block
constexpr int W = kOuterPanel;       // columns of a panel
constexpr int SUB = 16;              // sub-blocks of the triangular solves
// pitches of 4 (mod 16) doubles: the 4 x 4 elements that a half-warp of a DMMA
// fragment reads fall in 16 different pairs of banks
constexpr int PP = R + 4, VP = SUB + 4;
constexpr int NT = 512;
constexpr int VBLK = SUB * VP;       // one 16 x 16 inverse
constexpr int SLOT = kLuNB * kLuNB;  // doubles of a block's slot: inverses of the four U, then of the four L sub-blocks
constexpr size_t kSmem = (size_t)(W * PP + 2 * R * PP + 8 * VBLK + R) * 8 + 2 * R * 4 + 16;
constexpr int kSpin = 1 << 22;

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
// 16 bytes, of which the first `bytes` are read and the rest is zero
__device__ __forceinline__ void cp16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// waits for a pivot step's barrier, kStepTries at most, and adds the tries' bits to
// `late` (the caller goes on, with the identity as the row order; see step_status)
constexpr int kStepTries = 1 << 16;
__device__ __forceinline__ void wait_step(uint64_t* bar, int& late) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
  int i = 0;
  for (; i < kStepTries; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a)
        : "memory");
    if (ok) break;
  }
  late |= i;
  __syncwarp();
}
__device__ __forceinline__ void step_status(int late, int* status) {   // after a warp's last wait
  if (late & kStepTries) atomicOr(status, (int)DEV_TIMEOUT);
}

struct Smem {
  double (*P)[PP];      // [panel column][row]
  double (*Q)[R][PP];   // two 64 x 64 operands, [column][row]
  double* VU;           // inverses of the block's 16 x 16 U sub-blocks, [q][column][k]
  double* VL;           // of its L sub-blocks, [q][k][row]
  int* pr;              // physical row of each logical row (until the block is factored: the identity)
  int* lp;              // logical position of each step's pivot (the same)
  uint64_t* step;       // one barrier a pivot step: its column and pivot row are written
  int* stop;
};

// (cols x 64 rows) of the column-major A at (row0, col0) -> dst[column][row],
// zeros past `rows` rows and `cols` columns
__device__ __forceinline__ void load_block(double (*dst)[PP], const double* A, int64_t lda, int64_t row0, int rows,
                                           int64_t col0, int cols) {
  for (int e = threadIdx.x; e < R * (R / 2); e += NT) {
    const int c = e >> 5, r = (e & 31) * 2;
    const int b = c < cols ? max(0, min(2, rows - r)) * 8 : 0;
    cp16(&dst[c][r], b ? A + (col0 + c) * lda + row0 + r : A, b);
  }
}

// Inverses of the 16 x 16 triangles at logical rows and columns J0.. of D (row r
// of it is row rowof(r) of D), column i per lane, by columns so that a step is
// one FMA deep: the unit lower one to VL[q][k = column][row], the upper one to
// VU[q][column][k].
template <class RowOf>
__device__ __forceinline__ void inv_lower(Smem& s, double (*D)[PP], int J0, int lane, RowOf rowof) {
  double x[SUB];
#pragma unroll
  for (int r = 0; r < SUB; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < SUB - 1; ++k)
#pragma unroll
    for (int r = k + 1; r < SUB; ++r) x[r] = fma(-D[J0 + k][rowof(J0 + r)], x[k], x[r]);
  if (lane < SUB) {
    double* o = s.VL + (J0 / SUB) * VBLK + lane * VP;
#pragma unroll
    for (int r = 0; r < SUB; ++r) o[r] = x[r];
  }
}
template <class RowOf>
__device__ __forceinline__ void inv_upper(Smem& s, double (*D)[PP], int J0, int lane, RowOf rowof) {
  const double d = D[J0 + (lane & 15)][rowof(J0 + (lane & 15))];
  const double rd = d != 0.0 ? __drcp_rn(d) : 0.0;
  double x[SUB];
#pragma unroll
  for (int r = 0; r < SUB; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
  for (int k = SUB - 1; k >= 0; --k) {
    x[k] *= __shfl_sync(0xffffffffu, rd, k);
#pragma unroll
    for (int r = 0; r < k; ++r) x[r] = fma(-D[J0 + k][rowof(J0 + r)], x[k], x[r]);
  }
  if (lane < SUB) {
    double* o = s.VU + (J0 / SUB) * VBLK + lane * VP;
#pragma unroll
    for (int r = 0; r < SUB; ++r) o[r] = x[r];
  }
}

// The CTA factors the 64 x 64 diagonal block D ([column][row]) in place, rows
// never moving; last, D in logical row order, also to the matrix (Ad). Warp w
// holds columns 4 w .. 4 w + 3 in registers, lane l of it rows l and l + 32. It
// applies the pivots of the warps before it as they are published (the
// multipliers are D's column itself, the pivot's entries of its own columns
// come by shuffles), then makes its own four steps: so a step's chain, search
// -> multipliers -> next column -> its search, stays inside one warp and carries no
// other work. The pivot is LAPACK's: the largest |a| among the rows not yet
// taken, the first in logical order on ties. One warp for 16 columns with the
// products of the other columns between took 37 us a block.
__device__ __forceinline__ void factor_diag(Smem& s, double (*D)[PP], int nb, double* Ad, int64_t lda, int* status) {
  constexpr int C = R / (NT / 32);   // columns of a warp
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, own = warp * C;
  double a0[C], a1[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    a0[c] = D[own + c][lane];
    a1[c] = D[own + c][lane + 32];
  }
  bool used0 = false, used1 = false, zero = false;
  int late = 0;
  int pos0 = lane, pos1 = lane + 32;
  // the pivot row of step J takes logical place J, the row that had it the pivot's
  auto take = [&](int J, int pr, int lpos) {
    if (lane == pr) { used0 = true; pos0 = J; } else if (pos0 == J) { pos0 = lpos; }
    if (lane + 32 == pr) { used1 = true; pos1 = J; } else if (pos1 == J) { pos1 = lpos; }
  };
#pragma unroll 1
  for (int J = 0; J < own; ++J) {
    wait_step(s.step + J, late);
    const int pr = s.pr[J], src = pr & 31;
    const double l0 = D[J][lane], l1 = D[J][lane + 32];
    take(J, pr, s.lp[J]);
    const double m0 = used0 ? 0.0 : l0, m1 = used1 ? 0.0 : l1;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const double p = __shfl_sync(0xffffffffu, pr & 32 ? a1[c] : a0[c], src);
      a0[c] = fma(-m0, p, a0[c]);
      a1[c] = fma(-m1, p, a1[c]);
    }
  }
  // the search in column own + j: the lane's better row, the warp's largest high
  // word, the reciprocal of the lane's candidate
  bool second;
  unsigned hi, lo, mh;
  double rv;
  auto search = [&](double x0, double x1) {
    const unsigned long long k0 = used0 ? 0ull : (unsigned long long)__double_as_longlong(fabs(x0)) + 1ull;
    const unsigned long long k1 = used1 ? 0ull : (unsigned long long)__double_as_longlong(fabs(x1)) + 1ull;
    second = k1 > k0 || (k1 == k0 && pos1 < pos0);
    hi = (unsigned)((second ? k1 : k0) >> 32);
    lo = (unsigned)(second ? k1 : k0);
    mh = __reduce_max_sync(0xffffffffu, hi);
    rv = newton_rcp(second ? x1 : x0);
  };
  search(a0[0], a1[0]);
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const int J = own + j;
    const int pos = second ? pos1 : pos0;
    double v[C];   // the lane's candidate's entries from column J on
#pragma unroll
    for (int c = j; c < C; ++c) v[c] = second ? a1[c] : a0[c];
    const bool odd = !(fabs(v[j]) >= 0x1p-1000 && fabs(v[j]) <= 0x1p1000);
    const unsigned sec = __ballot_sync(0xffffffffu, second), odds = __ballot_sync(0xffffffffu, odd);
    unsigned win = __ballot_sync(0xffffffffu, hi == mh);
    if ((win & (win - 1)) | (win & odds)) {   // several lanes share the high word, or newton_rcp does not reach
      const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
      const bool top = hi == mh && lo == ml;
      const unsigned first = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : ~0u);
      win = __ballot_sync(0xffffffffu, top && (unsigned)pos == first);
      if (odd) rv = v[j] != 0.0 ? __drcp_rn(v[j]) : 0.0;
    }
    const int src = __ffs(win) - 1;
    const int pr = src + ((sec >> src) & 1) * 32;
    const double rp = __shfl_sync(0xffffffffu, rv, src);
    double p[C];
#pragma unroll
    for (int c = j + 1; c < C; ++c) p[c] = __shfl_sync(0xffffffffu, v[c], src);
    const int lpos = __shfl_sync(0xffffffffu, pos, src);
    take(J, pr, lpos);
    zero |= J < nb && rp == 0.0;
    // multipliers; zero for rows already taken, which the updates then leave alone
    const double m0 = used0 ? 0.0 : a0[j] * rp, m1 = used1 ? 0.0 : a1[j] * rp;
#pragma unroll
    for (int c = j + 1; c < C; ++c) {
      a0[c] = fma(-m0, p[c], a0[c]);
      a1[c] = fma(-m1, p[c], a1[c]);
    }
    // column J is final: U in the rows taken, L in the others
    const double f0 = used0 ? a0[j] : m0, f1 = used1 ? a1[j] : m1;
    if (j + 1 < C) search(a0[j + 1 < C ? j + 1 : 0], a1[j + 1 < C ? j + 1 : 0]);   // before the stores: the chain waits for it
    D[J][lane] = f0;
    D[J][lane + 32] = f1;
    if (lane == 0) {
      s.pr[J] = pr;
      s.lp[J] = lpos;
    }
    __syncwarp();
    if (lane == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(s.step + J))
                   : "memory");
  }
  if (zero && lane == 0) atomicOr(status, (int)DEV_ZERO_PIVOT);
  // the inverses of the sub-blocks, as each is done
  if (warp < 8) {
    const int J0 = (warp >> 1) * SUB;
    wait_step(s.step + J0 + SUB - 1, late);
    auto rowof = [&](int r) { return s.pr[r]; };
    if (warp & 1) inv_upper(s, D, J0, lane, rowof);
    else inv_lower(s, D, J0, lane, rowof);
  }
  step_status(late, status);
  __syncthreads();
  double (*L)[PP] = s.Q[0];
  for (int e = tid; e < R * R; e += NT) {
    const int col = e >> 6, r = e & 63;
    const double x = D[col][s.pr[r]];
    L[col][r] = x;
    if (r < nb && col < nb) Ad[col * lda + r] = x;
  }
  __syncthreads();
  for (int e = tid; e < R * R; e += NT) D[e >> 6][e & 63] = L[e >> 6][e & 63];
}

// C[64 columns][64 rows] -= X Q with X = 64 columns of the panel ([k][row]) and
// Q [column][k]: 16 warps, 16 x 16 each
__device__ __forceinline__ void update(double (*C)[PP], double (*X)[PP], double (*Q)[PP]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = (warp & 3) * 16, c0 = (warp >> 2) * 16;
  double d[2][2][2] = {};
#pragma unroll 4
  for (int k = 0; k < R; k += 4) {
    const double a0 = X[k + t][r0 + g], a1 = X[k + t][r0 + 8 + g];
    const double b0 = Q[c0 + g][k + t], b1 = Q[c0 + 8 + g][k + t];
    dmma(d[0][0][0], d[0][0][1], a0, b0);
    dmma(d[0][1][0], d[0][1][1], a0, b1);
    dmma(d[1][0][0], d[1][0][1], a1, b0);
    dmma(d[1][1][0], d[1][1][1], a1, b1);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) C[c0 + 8 * j + 2 * t + e][r0 + 8 * i + g] -= d[i][j][e];
}

// X (64 columns of the panel, [column][row]) <- X U^-1 by 16-column sub-blocks:
// U in Q ([column][k]), the inverses of its diagonal sub-blocks in VU. Eight
// warps, an 8-row tile each, which depends on no other (no barriers). Returns
// max|X|. A sub-block's solution by its inverse is refined once: without that its
// error grows with the sub-block's condition, to 7e-14 of |L||U| where the rows of a
// block differ by 1e6 in size and pivots are small (by substitution, and so, under
// 1e-15). 480 unknowns 0.490 -> 0.494 ms, 1,840 1.626 -> 1.651, 6,300 9.47 -> 9.53.
__device__ __forceinline__ double solve_l21(double (*X)[PP], double (*Q)[PP], const double* VU) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (warp >= 8) return 0.0;
  const int row = warp * 8 + g;
  double mx = 0.0;
#pragma unroll 1
  for (int q = 0; q < R / SUB; ++q) {
    const int c = q * SUB;
    double d[2][2][2] = {};   // [half][chain]
#pragma unroll 2
    for (int k = 0; k < c; k += 8)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double a = X[k + 4 * i + t][row];
#pragma unroll
        for (int h = 0; h < 2; ++h) dmma(d[h][i][0], d[h][i][1], a, Q[c + 8 * h + g][k + 4 * i + t]);
      }
    double b[2][2], x[2][2];   // the right-hand side and its solution
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        b[h][e] = X[c + 8 * h + 2 * t + e][row] - (d[h][0][e] + d[h][1][e]);
        X[c + 8 * h + 2 * t + e][row] = b[h][e];
        x[h][e] = 0.0;
      }
    __syncwarp();
    // x = b inv(U), then once x += (b - x U) inv(U)
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      double z[2][2][2] = {};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double a = X[c + 4 * k + t][row];
#pragma unroll
        for (int h = 0; h < 2; ++h) dmma(z[h][k & 1][0], z[h][k & 1][1], a, VU[q * VBLK + (8 * h + g) * VP + 4 * k + t]);
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          x[h][e] += z[h][0][e] + z[h][1][e];
          X[c + 8 * h + 2 * t + e][row] = x[h][e];
        }
      __syncwarp();
      if (pass == 1) break;
      double u[2][2][2] = {};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double a = X[c + 4 * k + t][row];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double w = 4 * k + t <= 8 * h + g ? Q[c + 8 * h + g][c + 4 * k + t] : 0.0;   // U alone: L lies below
          dmma(u[h][k & 1][0], u[h][k & 1][1], a, w);
        }
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) X[c + 8 * h + 2 * t + e][row] = b[h][e] - (u[h][0][e] + u[h][1][e]);
      __syncwarp();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) mx = fmax(mx, fabs(x[h][e]));
  }
  return mx;
}

// Y (columns [column][row], logical rows) <- L^-1 Y by 16-row sub-blocks, the 8
// columns y0.. of one warp: L [k][row], the inverses of its sub-blocks in VL
template <int YP>
__device__ __forceinline__ void solve_u12(double (*Y)[YP], int y0, int row0, double (*L)[PP], const double* VL) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double* y = Y[y0 + g] + row0;
  double* o[2] = {Y[y0 + 2 * t] + row0, Y[y0 + 2 * t + 1] + row0};
#pragma unroll 1
  for (int q = 0; q < R / SUB; ++q) {
    const int r = q * SUB;
    double d[2][2][2] = {};
#pragma unroll 2
    for (int k = 0; k < r; k += 8)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double b = y[k + 4 * i + t];
#pragma unroll
        for (int h = 0; h < 2; ++h) dmma(d[h][i][0], d[h][i][1], L[k + 4 * i + t][r + 8 * h + g], b);
      }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) o[e][r + 8 * h + g] -= d[h][0][e] + d[h][1][e];
    __syncwarp();
    double z[2][2][2] = {};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double b = y[r + 4 * k + t];
#pragma unroll
      for (int h = 0; h < 2; ++h) dmma(z[h][k & 1][0], z[h][k & 1][1], VL[q * VBLK + (4 * k + t) * VP + 8 * h + g], b);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) o[e][r + 8 * h + g] = z[h][0][e] + z[h][1][e];
    __syncwarp();
  }
}

// The panel at K0 (w columns, all rows below). CTA c (by ticket, so that a CTA
// waits only for CTAs already running) owns rows K0 + 64 c ..; CTA c < nblk
// factors diagonal block c and forms its rows of U. For each block b < c:
//   wait for block b's factors; L21 = A21 U11^-1; for each column block j > b:
//   wait for block b's U12 there, update.
// Block b's flag counts up: epoch base + 1 with its factors, + 1 with each column
// block of U12 written. What bounds it: the chain diagonal block -> L21 of
// the next 64 rows -> their update -> next diagonal block, on one SM each.
__global__ void __launch_bounds__(NT, 1)
k_panel64(double* __restrict__ A, int64_t lda, int64_t n, int64_t K0, int w, int32_t* __restrict__ ipiv,
          int* __restrict__ status, float* __restrict__ cert, double* __restrict__ slots, int* __restrict__ rowat,
          unsigned* __restrict__ sync, unsigned ticket0, unsigned flag0) {
  extern __shared__ __align__(16) unsigned char smem[];
  Smem s;
  double* p = reinterpret_cast<double*>(smem);
  s.P = reinterpret_cast<double (*)[PP]>(p); p += W * PP;
  s.Q = reinterpret_cast<double (*)[R][PP]>(p); p += 2 * R * PP;
  s.VU = p; p += 4 * VBLK;
  s.VL = p; p += 4 * VBLK;
  s.step = reinterpret_cast<uint64_t*>(p); p += R;
  s.pr = reinterpret_cast<int*>(p);
  s.lp = s.pr + R;
  s.stop = s.lp + R;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < R)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(s.step + tid)) : "memory");
  if (tid == 0) {
    s.lp[0] = (int)(atomicAdd(sync, 1u) - ticket0);
    *s.stop = 0;
  }
  __syncthreads();
  const int c = s.lp[0];
  __syncthreads();
  if (tid < R) s.pr[tid] = s.lp[tid] = tid;   // what a CTA that gives up leaves as its row order and pivots
  const int64_t r0 = K0 + (int64_t)c * R;
  const int rows = (int)imin64(R, n - r0);
  const int nblk = (w + R - 1) / R;
  volatile unsigned* flags = sync + 1;
#pragma unroll 1
  for (int j = 0; j < 4; ++j) {
    if (j < nblk) load_block(s.P + j * R, A, lda, r0, rows, K0 + j * R, w - j * R);
    cp_commit();
  }
  if (c == 0) cp_wait<3>(); else cp_wait<0>();
  __syncthreads();
  double lmax = 0.0;

  // waits until block b has published `level` (bounded); false: give up
  auto wait_flag = [&](int b, unsigned level) -> bool {
    if (tid == 0) {
      int i = 0;
      while ((int)(flags[b] - (flag0 + level)) < 0 && ++i < kSpin) {}
      if (i >= kSpin) { *s.stop = 1; atomicOr(status, (int)DEV_TIMEOUT); }
      __threadfence();
    }
    __syncthreads();
    return *s.stop == 0;
  };
  auto publish = [&](unsigned level) {   // this CTA's stores, then its flag
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      flags[c] = flag0 + level;
    }
  };
  // factor this CTA's diagonal block and publish it
  auto diagonal = [&]() {
    double (*D)[PP] = s.P + c * R;
    const int nb = rows;
    if (nb < R) {   // past the matrix: a unit diagonal
      for (int e = tid; e < R * R; e += NT)
        if ((e & 63) >= nb) D[e >> 6][e & 63] = (e >> 6) == (e & 63) ? 1.0 : 0.0;
      __syncthreads();
    }
    factor_diag(s, D, nb, A + r0 * lda + r0, lda, status);
    __syncthreads();
    double* slot = slots + (size_t)c * SLOT;
    for (int e = tid; e < 4 * SUB * SUB; e += NT) {
      const int q = e >> 8, i = (e >> 4) & 15, k = e & 15;
      slot[e] = s.VU[q * VBLK + i * VP + k];
      slot[4 * SUB * SUB + e] = s.VL[q * VBLK + i * VP + k];
    }
    publish(1);
  };
  // what no other CTA waits for: the pivots, and the rows left of the block in their order
  auto rest = [&]() {
    if (tid < R) {
      rowat[c * R + tid] = s.pr[tid];
      if (tid < rows) ipiv[r0 + tid] = (int32_t)(r0 + s.lp[tid]);
    }
    for (int e = tid; e < c * R * R; e += NT) {
      const int col = e >> 6, r = e & 63;
      if (r < rows) A[(K0 + col) * lda + r0 + r] = s.P[col][s.pr[r]];
    }
  };
  // this CTA's rows of U in column block j, from its updated rows
  auto u12 = [&](int j, double (*Y)[PP]) {
    __syncthreads();
    for (int e = tid; e < R * R; e += NT) Y[e >> 6][e & 63] = s.P[j * R + (e >> 6)][s.pr[e & 63]];
    __syncthreads();
    if (tid < 256) solve_u12<PP>(Y, (tid >> 5) * 8, 0, s.P + c * R, s.VL);
    __syncthreads();
    for (int e = tid; e < R * R; e += NT) {
      const int col = e >> 6, r = e & 63;
      if (r < rows && j * R + col < w) A[(K0 + j * R + col) * lda + r0 + r] = Y[col][r];
    }
    publish(1 + j - c);
  };

  if (c == 0) {
    diagonal();
    cp_wait<0>();
    for (int j = 1; j < nblk; ++j) u12(j, s.Q[j & 1]);
    rest();
    return;
  }
  const int steps = min(c, nblk);
#pragma unroll 1
  for (int b = 0; b < steps; ++b) {
    if (!wait_flag(b, 1)) break;
    const int64_t k0 = K0 + b * R;
    load_block(s.Q[0], A, lda, k0, R, k0, R);
    for (int e = tid; e < 4 * SUB * SUB; e += NT)
      s.VU[(e >> 8) * VBLK + ((e >> 4) & 15) * VP + (e & 15)] = __ldcg(slots + (size_t)b * SLOT + e);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    lmax = fmax(lmax, solve_l21(s.P + b * R, s.Q[0], s.VU));
    bool ok = true;
#pragma unroll 1
    for (int j = b + 1; j < nblk; ++j) {
      ok = wait_flag(b, 1 + j - b);   // its barrier also ends the reads of Q from two blocks back
      if (!ok) break;
      double (*Q)[PP] = s.Q[(j - b) & 1];
      load_block(Q, A, lda, k0, R, K0 + j * R, w - j * R);
      cp_commit();
      cp_wait<0>();
      __syncthreads();
      update(s.P + j * R, s.P + b * R, Q);
      if (b == c - 1) {
        __syncthreads();
        if (j == c) diagonal();
        else u12(j, Q);
      }
    }
    if (!ok) break;
    __syncthreads();
  }
  if (c < nblk)
    rest();
  else   // rows below the panel's blocks: L21
    for (int e = tid; e < nblk * R * R; e += NT) {
      const int col = e >> 6, r = e & 63;
      if (r < rows && col < w) A[(K0 + col) * lda + r0 + r] = s.P[col][r];
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
  if (lane == 0 && lmax > 0.0) atomicMax(reinterpret_cast<int*>(cert), __float_as_int((float)lmax));
}

// ----------------------------------------------------------------------------
// Columns beside a factored panel of 256 columns and rows: on [cl0, cl1) each
// block's rows in their logical order; on [cr0, cr1) also U12, 16 columns a CTA,
// by blocks: U_b = L_bb^-1 Y_b (16-row sub-blocks with the stored inverses), then
// the blocks below less L_b'b U_b. The ten 64 x 64 blocks of L stream through
// two buffers.
namespace strip {
constexpr int COLS = 16, NT = 256, XP = W + 4;   // XP = 4 (mod 16)
constexpr size_t kSmem = (size_t)(COLS * XP + 2 * R * PP + 4 * VBLK) * 8 + W;   // two CTAs an SM
}  // namespace strip

__global__ void __launch_bounds__(strip::NT, 2)
k_strip64(double* __restrict__ A, int64_t lda, int64_t K0, int w, const double* __restrict__ slots,
          const int* __restrict__ rowat, int64_t cl0, int64_t cl1, int64_t cr0, int64_t cr1) {
  using namespace strip;
  constexpr int NT = strip::NT;
  extern __shared__ __align__(16) unsigned char smem[];
  double (*X)[XP] = reinterpret_cast<double (*)[XP]>(smem);
  double (*L)[R][PP] = reinterpret_cast<double (*)[R][PP]>(smem + (size_t)COLS * XP * 8);
  double* V = reinterpret_cast<double*>(smem + (size_t)(COLS * XP + 2 * R * PP) * 8);   // the block's inverses, [q][k][row]
  uint8_t* ra = reinterpret_cast<uint8_t*>(V + 4 * VBLK);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int64_t gl = (cl1 - cl0 + COLS - 1) / COLS;
  const bool right = (int64_t)blockIdx.x >= gl;
  const int64_t c0 = right ? cr0 + ((int64_t)blockIdx.x - gl) * COLS : cl0 + (int64_t)blockIdx.x * COLS;
  const int nc = (int)imin64(COLS, (right ? cr1 : cl1) - c0);
  const int nblk = (w + R - 1) / R;
  auto stage = [&](int i, int b2, int b) {   // L(b2, b) into buffer i; only whole panels have columns to the right
    for (int e = tid; e < R * (R / 2); e += NT) {
      const int k = e >> 5, r = (e & 31) * 2;
      cp16(&L[i][k][r], A + (K0 + b * R + k) * lda + K0 + b2 * R + r, 16);
    }
    if (b2 == b)   // the last use of V was before the previous block's last product
      for (int e = tid; e < 4 * SUB * SUB / 2; e += NT)
        cp16(V + (e >> 3) * VP + (e & 7) * 2, slots + (size_t)b * SLOT + 4 * SUB * SUB + 2 * e, 16);
    cp_commit();
  };
  if (right) stage(0, 0, 0);
  for (int e = tid; e < w; e += NT) ra[e] = (uint8_t)rowat[e];
  __syncthreads();
  // the rows in logical order
  for (int e = tid; e < COLS * W; e += NT) {
    const int col = e >> 8, r = e & 255;
    X[col][r] = (col < nc && r < w) ? A[(c0 + col) * lda + K0 + (r & ~63) + ra[r]] : 0.0;
  }
  __syncthreads();
  if (!right) {
    for (int e = tid; e < COLS * W; e += NT) {
      const int col = e >> 8, r = e & 255;
      if (col < nc && r < w && ra[r] != (r & 63)) A[(c0 + col) * lda + K0 + r] = X[col][r];
    }
    return;
  }
  int i = 0;
#pragma unroll 1
  for (int b = 0; b < nblk; ++b)
#pragma unroll 1
    for (int b2 = b; b2 < nblk; ++b2, ++i) {
      const int nb = b2 + 1 < nblk ? b : b + 1, nb2 = b2 + 1 < nblk ? b2 + 1 : b + 1;
      if (nb < nblk) { stage((i + 1) & 1, nb2, nb); cp_wait<1>(); } else { cp_wait<0>(); }
      __syncthreads();
      double (*Lb)[PP] = L[i & 1];
      if (b2 == b) {   // U_b, an 8-column tile a warp
        if (warp < COLS / 8) solve_u12<XP>(X, warp * 8, b * R, Lb, V);
      } else {   // X_b2 -= L(b2, b) U_b: a row tile a warp, both column tiles
        const int r = warp * 8 + g;
        double d[2][2] = {};
#pragma unroll 4
        for (int k = 0; k < R; k += 4) {
          const double a = Lb[k + t][r];
          dmma(d[0][0], d[0][1], a, X[g][b * R + k + t]);
          dmma(d[1][0], d[1][1], a, X[8 + g][b * R + k + t]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) X[8 * j + 2 * t + e][b2 * R + r] -= d[j][e];
      }
      __syncthreads();
    }
  for (int e = tid; e < COLS * W; e += NT) {
    const int col = e >> 8, r = e & 255;
    if (col < nc && r < w) A[(c0 + col) * lda + K0 + r] = X[col][r];
  }
}

}  // namespace p64

// Two streams share the work of each panel P:
//  * c->stream (high priority, the critical path): the panel, then, once the
//    previous panel's trailing update is done, P's swaps and U12 in the next
//    panel's columns and the update of those columns;
//  * c->stream2: the swaps left of P, U12 and the update beyond the next panel.
// Row swaps stay inside 64-row blocks, so the swaps of different blocks
// commute, and a row update commutes with a swap of the rows of both C and L.
//
// The update's products stay in FP64: as seven INT8 digits under a scale a row and
// column (exact sums on the INT8 tensor cores) it took 31 ms of a factorisation of
// 12,000 where this takes 47, but an entry loses the bits by which it lies below its
// row's largest. The factors' error was 1e-9 of |L||U| in places (here 4e-15), and
// the response of one of two bodies to the other held 9 digits instead of 15.
template <>
int lu_factor<double>(fp_ctx* c, double* A, int64_t n, int64_t lda, int32_t* ipiv, float* cert) {
  constexpr int W = p64::W, R = p64::R;
  if (((reinterpret_cast<uintptr_t>(A) | (uintptr_t)(lda * 8)) & 15) != 0)
    return c->err.set(FP_EINVAL, "lu_factor: the matrix must be 16-byte aligned with an even leading dimension");
  FP_CUDA_TRY(c->err, cudaMemsetAsync(cert, 0, sizeof(float), c->stream));
  static SmemAttr attr_panel, attr_strip;
  FP_CUDA_TRY(c->err, attr_panel.ensure(p64::k_panel64, (int)p64::kSmem));
  FP_CUDA_TRY(c->err, attr_strip.ensure(p64::k_strip64, (int)p64::strip::kSmem));
  static_assert(W / R <= kPanelSlots && 8 * p64::SUB * p64::SUB <= p64::SLOT, "one scratch slot per block of a panel");
  // the blocks' inverses and row orders, two sets (panel parity): stream2's
  // strip of panel P reads its set while panel P + 1 fills the other
  double* const slots0 = reinterpret_cast<double*>(c->d_minv);
  int* const rowat0 = reinterpret_cast<int*>(reinterpret_cast<char*>(c->d_minv) + kMinvBytes);
  auto at = [&](int64_t r, int64_t col) { return A + col * lda + r; };
  c->trace.base = tr_event(c);
  // stream2 starts after everything already queued on c->stream
  FP_CUDA_TRY(c->err, cudaEventRecord(c->ev_rest, c->stream));
  FP_CUDA_TRY(c->err, cudaStreamWaitEvent(c->stream2, c->ev_rest, 0));
  for (int64_t K0 = 0; K0 < n; K0 += W) {
    const int64_t kend = std::min<int64_t>(K0 + W, n);
    const int64_t knext = std::min<int64_t>(kend + W, n);   // next panel: columns [kend, knext)
    const int set = (int)((K0 / W) & 1), w = (int)(kend - K0);
    double* const slots = slots0 + (size_t)set * kPanelSlots * p64::SLOT;
    int* const rowat = rowat0 + (size_t)set * kPanelSlots * R;
    {
      const unsigned ctas = (unsigned)((n - K0 + R - 1) / R);
      TraceScope tr(c, TR_L21);
      p64::k_panel64<<<ctas, p64::NT, p64::kSmem, c->stream>>>(A, lda, n, K0, w, ipiv, c->d_status, cert, slots, rowat,
                                                              c->d_p64, c->p64_ticket, c->p64_flag);
      ++c->nlaunch;
      FP_CUDA_TRY(c->err, cudaGetLastError());
      c->p64_ticket += ctas;
      c->p64_flag += 8;   // more than the levels a block publishes
    }
    FP_CUDA_TRY(c->err, cudaEventRecord(c->ev_panel, c->stream));
    auto strip = [&](int64_t cl0, int64_t cl1, int64_t cr0, int64_t cr1) -> int {
      const int64_t g = (cl1 - cl0 + p64::strip::COLS - 1) / p64::strip::COLS +
                        (cr1 - cr0 + p64::strip::COLS - 1) / p64::strip::COLS;
      if (g <= 0) return FP_OK;
      TraceScope tr(c, TR_STRIP);
      p64::k_strip64<<<(unsigned)g, p64::strip::NT, p64::strip::kSmem, c->stream>>>(A, lda, K0, w, slots, rowat, cl0, cl1,
                                                                                   cr0, cr1);
      ++c->nlaunch;
      FP_CUDA_TRY(c->err, cudaGetLastError());
      return FP_OK;
    };
    // columns [c0, c1) right of the panel -= L21 U12
    auto update = [&](int64_t c0, int64_t c1) -> int {
      return gemm_sub_f64(c, at(kend, K0), at(K0, c0), at(kend, c0), lda, n - kend, c1 - c0, w);
    };
    if (knext > kend) {
      FP_CUDA_TRY(c->err, cudaStreamWaitEvent(c->stream, c->ev_rest, 0));
      if (int rc = strip(0, 0, kend, knext)) return rc;
      if (int rc = update(kend, knext)) return rc;
    }
    {
      OnStream2 on2(c);
      FP_CUDA_TRY(c->err, cudaStreamWaitEvent(c->stream, c->ev_panel, 0));
      if (int rc = strip(0, K0, knext, n)) return rc;
      if (n > knext)
        if (int rc = update(knext, n)) return rc;
      FP_CUDA_TRY(c->err, cudaEventRecord(c->ev_rest, c->stream));
    }
  }
  // join: c->stream continues after the last work on stream2
  FP_CUDA_TRY(c->err, cudaStreamWaitEvent(c->stream, c->ev_rest, 0));
  return FP_OK;
}

}  // namespace fpb
