// FP64 LU of the FP64 form: 256-column panels in 64-column blocks, partial
// pivoting inside each 64 x 64 diagonal block (the certificate max|L21| <= 1
// says that every pivot is the one LAPACK's dgetrf picks; see fp_lu.cu).
//
// Per panel: k_panel64 factors its columns in one launch; k_strip64 swaps the
// panel's rows and forms U12 in the columns beside it; the trailing update
// follows on the INT8 tensor cores (fp_i8.cu) or the FP64 tensor path
// (fp_lu.cu), the next panel's columns first.
//
// The panel is a chain of 256 dependent pivot steps, so its kernels are built
// for latency: one CTA of 16 warps holds 64 rows of the panel in shared memory
// for the whole panel, and blocks hand each other their factors through L2. One
// launch per 64 columns, with the rows reloaded each time and SIMT products,
// took 490 us a panel (strip and next-panel update included) where this takes
// 240; factorisation of 480 unknowns 0.95 -> 0.60 ms, 1,840 3.47 -> 1.96,
// 6,300 14.8 -> 8.5, 12,000 43.1 -> 33.4 ms.
#include "fp_internal.cuh"

namespace fpb {
namespace p64 {

constexpr int R = 64;                // rows of a CTA, columns of a block
constexpr int W = kOuterPanel;       // columns of a panel
constexpr int SUB = 16;              // columns factored by one warp at a time
// pitches of 4 (mod 16) doubles: the 4 x 4 elements that a half-warp of a DMMA
// fragment reads fall in 16 different pairs of banks
constexpr int PP = R + 4, VP = SUB + 4;
constexpr int NT = 512;
constexpr int VBLK = SUB * VP;       // one 16 x 16 inverse
constexpr int SLOT = kLuNB * kLuNB;  // doubles of a block's slot: inverses of the four U, then of the four L sub-blocks
constexpr size_t kSmem = (size_t)(W * PP + 2 * R * PP + 8 * VBLK + 2 * SUB) * 8 + 2 * R * 4 + 64;
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
__device__ __forceinline__ void pair_bar(int warp) {   // the two warps 2 i, 2 i + 1
  asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
}

struct Smem {
  double (*P)[PP];      // [panel column][row]
  double (*Q)[R][PP];   // two 64 x 64 operands, [column][row]
  double* VU;           // inverses of the block's 16 x 16 U sub-blocks, [q][column][k]
  double* VL;           // of its L sub-blocks, [q][k][row]
  double* pv;           // the pivot row of a step, two copies
  int* pr;              // physical row of each logical row
  int* lp;              // logical position of each step's pivot
  unsigned long long* used;   // rows taken as pivots after each sub-block, two copies
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

// Columns J0 .. J0 + 15 of the diagonal block D ([column][row], 64 rows) by one
// warp: lane l holds rows l and l + 32, their entries shifted so that a[0] is
// the current column (a rolled loop: the code stays in the instruction cache).
// The pivot is LAPACK's: the largest |a| among the rows not yet taken, the
// first in logical order on ties. Each lane forms the reciprocals of its
// own candidates while the search runs.
__device__ __forceinline__ void factor_sub(Smem& s, double (*D)[PP], int J0, int nb, bool& used0, bool& used1, int& pos0,
                                           int& pos1, bool& zero) {
  const int lane = threadIdx.x & 31;
  double a0[SUB], a1[SUB];
#pragma unroll
  for (int c = 0; c < SUB; ++c) {
    a0[c] = D[J0 + c][lane];
    a1[c] = D[J0 + c][lane + 32];
  }
#pragma unroll 1
  for (int j = 0; j < SUB; ++j) {
    const int J = J0 + j;
    double* const pv = s.pv + (j & 1) * SUB;
    const unsigned long long k0 = used0 ? 0ull : (unsigned long long)__double_as_longlong(fabs(a0[0])) + 1ull;
    const unsigned long long k1 = used1 ? 0ull : (unsigned long long)__double_as_longlong(fabs(a1[0])) + 1ull;
    const bool second = k1 > k0 || (k1 == k0 && pos1 < pos0);
    const unsigned long long k = second ? k1 : k0;
    const int pos = second ? pos1 : pos0;
    const double r0 = a0[0] != 0.0 ? __drcp_rn(a0[0]) : 0.0, r1 = a1[0] != 0.0 ? __drcp_rn(a1[0]) : 0.0;
    const unsigned hi = (unsigned)(k >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == mh ? (unsigned)k : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    const bool top = hi == mh && (unsigned)k == ml;
    const unsigned lead = __reduce_min_sync(0xffffffffu, top ? (unsigned)((pos << 6) | (second ? 32 : 0) | lane) : ~0u);
    const int src = lead & 31, lpos = (int)(lead >> 6);
    const bool mine = lane == src, psec = (lead >> 5) & 1;
    if (mine) {   // the pivot row to all lanes
      double2* o = reinterpret_cast<double2*>(pv);
#pragma unroll
      for (int c = 0; c < SUB; c += 2) o[c / 2] = psec ? make_double2(a1[c], a1[c + 1]) : make_double2(a0[c], a0[c + 1]);
    }
    const double rp = __shfl_sync(0xffffffffu, psec ? r1 : r0, src);
    const double p1 = __shfl_sync(0xffffffffu, psec ? a1[1] : a0[1], src);
    zero |= J < nb && rp == 0.0;
    // the pivot row takes logical place J, the row that had it the pivot's
    if (mine && !psec) { used0 = true; pos0 = J; } else if (pos0 == J) { pos0 = lpos; }
    if (mine && psec) { used1 = true; pos1 = J; } else if (pos1 == J) { pos1 = lpos; }
    if (lane == 0) {
      s.pr[J] = src + (psec ? 32 : 0);
      s.lp[J] = lpos;
    }
    // multipliers; zero for rows already taken, which the updates below then leave alone
    const double m0 = used0 ? 0.0 : a0[0] * rp, m1 = used1 ? 0.0 : a1[0] * rp;
    a0[0] = fma(-m0, p1, a0[1]);   // the next column first: its search waits for it
    a1[0] = fma(-m1, p1, a1[1]);
    if (!used0) D[J][lane] = m0;
    if (!used1) D[J][lane + 32] = m1;
    __syncwarp();
    double u[SUB];
    const double2* in = reinterpret_cast<const double2*>(pv);
#pragma unroll
    for (int c = 0; c < SUB; c += 2) {
      const double2 v = in[c / 2];
      u[c] = v.x;
      u[c + 1] = v.y;
    }
#pragma unroll
    for (int c = 1; c < SUB - 1; ++c) {
      a0[c] = fma(-m0, u[c + 1], a0[c + 1]);
      a1[c] = fma(-m1, u[c + 1], a1[c + 1]);
    }
    if (lane < SUB - j) D[J + lane][src + (psec ? 32 : 0)] = pv[lane];   // the pivot's row of U
  }
  const unsigned b0 = __ballot_sync(0xffffffffu, used0), b1 = __ballot_sync(0xffffffffu, used1);
  if (lane == 0) s.used[(J0 / SUB) & 1] = (unsigned long long)b1 << 32 | b0;
}

// inverse of the 16 x 16 unit lower (lane < 16) triangle of the logical rows
// and columns J0.. of D, column i per lane, to VL[q][k = column][row]
__device__ __forceinline__ void inv_lower(Smem& s, double (*D)[PP], int J0, int lane) {
  if (lane >= SUB) return;
  double x[SUB];
#pragma unroll
  for (int r = 0; r < SUB; ++r) {
    double v = r == lane ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < r; ++k) v = fma(-D[J0 + k][s.pr[J0 + r]], x[k], v);
    x[r] = v;
  }
  double* o = s.VL + (J0 / SUB) * VBLK + lane * VP;
#pragma unroll
  for (int r = 0; r < SUB; ++r) o[r] = x[r];
}
// inverse of the upper triangle, column i per lane, to VU[q][column][k]
__device__ __forceinline__ void inv_upper(Smem& s, double (*D)[PP], int J0, int lane) {
  if (lane >= SUB) return;
  double x[SUB];
#pragma unroll
  for (int r = SUB - 1; r >= 0; --r) {
    double v = r == lane ? 1.0 : 0.0;
#pragma unroll
    for (int k = SUB - 1; k > r; --k) v = fma(-D[J0 + k][s.pr[J0 + r]], x[k], v);
    const double d = D[J0 + r][s.pr[J0 + r]];
    x[r] = d != 0.0 ? v * __drcp_rn(d) : 0.0;
  }
  double* o = s.VU + (J0 / SUB) * VBLK + lane * VP;
#pragma unroll
  for (int r = 0; r < SUB; ++r) o[r] = x[r];
}

// The CTA factors the 64 x 64 diagonal block D in place, rows never moving:
// after each 16 columns the U rows of the columns right of them, then the
// rank-16 update of the rows not yet taken, the next 16 columns first, so that
// warp 0 goes on with them while the other warps finish. Last, D in logical
// row order.
__device__ __forceinline__ void factor_diag(Smem& s, double (*D)[PP], int nb, int* status) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  bool used0 = false, used1 = false, zero = false;
  int pos0 = lane, pos1 = lane + 32;
  // one 8 x 8 tile of the update of columns J1.. from the pivots J1 - 16 .. J1 - 1
  auto tile = [&](int J1, int ct, int rt) {
    const int row = rt * 8 + g, c0 = J1 + ct * 8;
    double d0 = 0.0, d1 = 0.0;
#pragma unroll
    for (int k = 0; k < SUB; k += 4)
      dmma(d0, d1, D[J1 - SUB + k + t][row], D[c0 + g][s.pr[J1 - SUB + k + t]]);
    if (!((s.used[(J1 / SUB - 1) & 1] >> row) & 1)) {
      D[c0 + 2 * t][row] -= d0;
      D[c0 + 2 * t + 1][row] -= d1;
    }
  };
#pragma unroll 1
  for (int q = 0; q < R / SUB; ++q) {
    const int J0 = q * SUB, J1 = J0 + SUB, right = (R - J1) / 8;   // column tiles right of the sub-block
    if (warp == 0) {
      factor_sub(s, D, J0, nb, used0, used1, pos0, pos1, zero);
    } else if (q > 0) {   // the columns beyond, of the previous step; the inverses of its sub-blocks
      for (int i = 16 + warp - 1; i < R - J0; i += 15) tile(J0, i >> 3, i & 7);
      if (warp == 14) inv_lower(s, D, J0 - SUB, lane);
      if (warp == 15) inv_upper(s, D, J0 - SUB, lane);
    }
    __syncthreads();
    if (right == 0) break;
    if (tid < R - J1) {   // U rows of this sub-block: a column per thread
      double* col = D[J1 + tid];
      double u[SUB];
#pragma unroll
      for (int k = 0; k < SUB; ++k) u[k] = col[s.pr[J0 + k]];
#pragma unroll
      for (int k = 0; k < SUB - 1; ++k)
#pragma unroll
        for (int r = k + 1; r < SUB; ++r) u[r] = fma(-D[J0 + k][s.pr[J0 + r]], u[k], u[r]);
#pragma unroll
      for (int k = 1; k < SUB; ++k) col[s.pr[J0 + k]] = u[k];
    }
    __syncthreads();
    tile(J1, warp >> 3, warp & 7);   // the next 16 columns
    __syncthreads();
  }
  if (warp == 0 && zero && lane == 0) atomicOr(status, (int)DEV_ZERO_PIVOT);
  if (warp == 14) inv_lower(s, D, R - SUB, lane);
  if (warp == 15) inv_upper(s, D, R - SUB, lane);
  double (*L)[PP] = s.Q[0];
  for (int e = tid; e < R * R; e += NT) L[e >> 6][e & 63] = D[e >> 6][s.pr[e & 63]];
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
// U in Q ([column][k]), the inverses of its diagonal sub-blocks in VU. Two
// warps an 8-row tile, 8 columns of a sub-block each. Returns max|X|.
__device__ __forceinline__ double solve_l21(double (*X)[PP], double (*Q)[PP], const double* VU) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int row = (warp >> 1) * 8 + g, half = (warp & 1) * 8;
  double mx = 0.0;
#pragma unroll 1
  for (int q = 0; q < R / SUB; ++q) {
    const int c = q * SUB + half;
    double d0 = 0.0, d1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll 2
    for (int k = 0; k < q * SUB; k += 8) {
      dmma(d0, d1, X[k + t][row], Q[c + g][k + t]);
      dmma(e0, e1, X[k + 4 + t][row], Q[c + g][k + 4 + t]);
    }
    X[c + 2 * t][row] -= d0 + e0;
    X[c + 2 * t + 1][row] -= d1 + e1;
    pair_bar(warp);
    double a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = X[q * SUB + 4 * k + t][row];
    d0 = d1 = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) dmma(d0, d1, a[k], VU[q * VBLK + (half + g) * VP + 4 * k + t]);
    pair_bar(warp);
    X[c + 2 * t][row] = d0;
    X[c + 2 * t + 1][row] = d1;
    mx = fmax(mx, fmax(fabs(d0), fabs(d1)));
    pair_bar(warp);
  }
  return mx;
}

// Y (64 columns, [column][row], logical rows) <- L^-1 Y by 16-row sub-blocks: L in
// the panel's columns ([k][row]), the inverses of its sub-blocks in VL. Two
// warps an 8-column tile, 8 rows of a sub-block each.
__device__ __forceinline__ void solve_u12(double (*Y)[PP], double (*L)[PP], const double* VL) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int c = (warp >> 1) * 8, half = (warp & 1) * 8;
#pragma unroll 1
  for (int q = 0; q < R / SUB; ++q) {
    const int r = q * SUB + half + g;
    double d0 = 0.0, d1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll 2
    for (int k = 0; k < q * SUB; k += 8) {
      dmma(d0, d1, L[k + t][r], Y[c + g][k + t]);
      dmma(e0, e1, L[k + 4 + t][r], Y[c + g][k + 4 + t]);
    }
    Y[c + 2 * t][r] -= d0 + e0;
    Y[c + 2 * t + 1][r] -= d1 + e1;
    pair_bar(warp);
    double b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] = Y[c + g][q * SUB + 4 * k + t];
    d0 = d1 = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) dmma(d0, d1, VL[q * VBLK + (4 * k + t) * VP + half + g], b[k]);
    pair_bar(warp);
    Y[c + 2 * t][r] = d0;
    Y[c + 2 * t + 1][r] = d1;
    pair_bar(warp);
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
  s.pv = p; p += 2 * SUB;
  s.used = reinterpret_cast<unsigned long long*>(p); p += 2;
  s.stop = reinterpret_cast<int*>(p); p += 1;
  s.pr = reinterpret_cast<int*>(p);
  s.lp = s.pr + R;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) {
    s.lp[0] = (int)(atomicAdd(sync, 1u) - ticket0);
    *s.stop = 0;
  }
  __syncthreads();
  const int c = s.lp[0];
  __syncthreads();
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
  // factor this CTA's diagonal block, write it and the rows left of it, publish
  auto diagonal = [&]() {
    double (*D)[PP] = s.P + c * R;
    const int nb = rows;
    if (nb < R) {   // past the matrix: a unit diagonal
      for (int e = tid; e < R * R; e += NT)
        if ((e & 63) >= nb) D[e >> 6][e & 63] = (e >> 6) == (e & 63) ? 1.0 : 0.0;
      __syncthreads();
    }
    factor_diag(s, D, nb, status);
    __syncthreads();
    for (int e = tid; e < R * R; e += NT) {
      const int col = e >> 6, r = e & 63;
      if (r < nb && col < nb) A[(r0 + col) * lda + r0 + r] = D[col][r];
    }
    double* slot = slots + (size_t)c * SLOT;
    for (int e = tid; e < 4 * SUB * SUB; e += NT) {
      const int q = e >> 8, i = (e >> 4) & 15, k = e & 15;
      slot[e] = s.VU[q * VBLK + i * VP + k];
      slot[4 * SUB * SUB + e] = s.VL[q * VBLK + i * VP + k];
    }
    publish(1);
    if (tid < R) {
      rowat[c * R + tid] = s.pr[tid];
      if (tid < nb) ipiv[r0 + tid] = (int32_t)(r0 + s.lp[tid]);
    }
    for (int e = tid; e < c * R * R; e += NT) {
      const int col = e >> 6, r = e & 63;
      if (r < nb) A[(K0 + col) * lda + r0 + r] = s.P[col][s.pr[r]];
    }
  };
  // this CTA's rows of U in column block j, from its updated rows
  auto u12 = [&](int j, double (*Y)[PP]) {
    __syncthreads();
    for (int e = tid; e < R * R; e += NT) Y[e >> 6][e & 63] = s.P[j * R + (e >> 6)][s.pr[e & 63]];
    __syncthreads();
    solve_u12(Y, s.P + c * R, s.VL);
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
  if (c >= nblk)   // rows below the panel's blocks: L21
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
      if (b2 == b) {   // U_b: warps 0..3, an 8-column tile each pair, 8 rows of a sub-block each
        if (warp < 4) {
          const int c = (warp >> 1) * 8, half = (warp & 1) * 8;
#pragma unroll 1
          for (int q = 0; q < R / SUB; ++q) {
            const int r = q * SUB + half + g;
            double* x0 = X[c + 2 * t] + b * R + r;
            double* x1 = X[c + 2 * t + 1] + b * R + r;
            const double* y = X[c + g] + b * R;
            double d0 = 0.0, d1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll 2
            for (int k = 0; k < q * SUB; k += 8) {
              dmma(d0, d1, Lb[k + t][r], y[k + t]);
              dmma(e0, e1, Lb[k + 4 + t][r], y[k + 4 + t]);
            }
            *x0 -= d0 + e0;
            *x1 -= d1 + e1;
            pair_bar(warp);
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = y[q * SUB + 4 * k + t];
            d0 = d1 = 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) dmma(d0, d1, V[q * VBLK + (4 * k + t) * VP + half + g], v[k]);
            pair_bar(warp);
            *x0 = d0;
            *x1 = d1;
            pair_bar(warp);
          }
        }
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
// Panels with kI8Rows rows below them update on the INT8 tensor cores
// (fp_i8.cu) unless a variant of FP_TUNE_FP64_DMMA is asked for. Below that
// the digits' two launches and a tile's latency (35 us) cost what the INT8
// update saves.
constexpr int64_t kI8Rows = 2048;

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
  const bool i8 = c->fp64_dmma == 6 && n >= W + kI8Rows;
  if (i8)
    if (int rc = i8_scratch(c, n)) return rc;
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
    const bool digits = i8 && n - kend >= kI8Rows;
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
    if (digits)
      if (int rc = i8_slice_rows(c, set, at(kend, K0), lda, n - kend)) return rc;
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
      if (digits) return i8_gemm_sub(c, set, at(K0, c0), at(kend, c0), lda, n - kend, c0 - kend, c1 - c0);
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
