// FP64 trailing update C -= A B of the FP64 factorisation on the INT8 tensor
// cores (tcgen05.mma kind::i8), by an error-free split of the operands into
// 8-bit digits (Ootomo, Ozaki & Yokota, "DGEMM on integer matrix
// multiplication unit", 2024):
//
//   row i of A:     a(i,k) = 2^(ea_i - 54) sum_s 256^(6-s) A_s(i,k)
//   column j of B:  b(k,j) = 2^(eb_j - 54) sum_t 256^(6-t) B_t(k,j)
//
// with |a(i,:)| < 2^ea_i and seven balanced digits in -128..127 (55 bits below
// the row's largest entry; an FP64 entry has 53). The products A_s B_t are
// exact in INT32 (256 terms of 2^14, at most 8 pairs: 2^25), those of one
// s + t share an accumulator, and those with s + t > 7 are left out: they lie
// under 2^-64 of the row's times the column's largest entry, below the
// rounding of an FP64 accumulation of K = 256 products. The eight
// accumulators are summed in FP64, smallest weight first, and subtracted from
// C with one rounding. Measured against a long-double factorisation, the
// residual |PA - LU| of AICs of wings and spheres (1,800 to 1,920 panels) is
// that of an FP64 product (3.4e-18 against 3.5e-18, 2.45e-18 for both); with
// s + t <= 6 it is 1.5 times larger, with six digits 250 times.
//
// Bounds: 34 digit products of 2 m n K operations on the INT8 pipe (about 4.5
// POP/s dense) against 2 m n K FP64 operations on the FP64 tensor path (37.2
// TFLOP/s): a ceiling 3.5 times higher.
#include <type_traits>

#include "fp_internal.cuh"
#include "fp_umma.cuh"

namespace fpb {
namespace i8 {
using namespace tc;

constexpr int S = 7, G = 8;             // digits of an operand, sums s + t
constexpr int BM = 128, BN = 128;       // output tile
constexpr int PG = 4;                   // sums of a pass: PG * BN = 512 TMEM columns
constexpr int KB = 64, STAGES = 2;      // K block of a stage: rows of 64 bytes (64-byte swizzle)
constexpr int KP = kOuterPanel;         // K of an operand
constexpr int NK = KP / KB;
constexpr int DIG = BM * KB;            // bytes of one digit of an operand's K block
constexpr int BLOCK = S * DIG, STAGE = 2 * BLOCK;
constexpr int SMEM = STAGES * STAGE + 1024 + 256;
constexpr int EPI_WARPS = 8, THREADS = 32 * (2 + EPI_WARPS);
// D s32 (2), A and B signed 8-bit (1), both K-major, N >> 3, M >> 4
constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// K-major descriptor of rows of KB = 64 bytes, 64-byte swizzle (layout 4),
// SBO = 8 rows, version 1
__device__ __forceinline__ uint64_t sdesc64(uint32_t addr) {
  uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)((8u * KB) >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)4u << 61;
  return d;
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(IDESC), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
// exact FP64 value of an INT32 without the conversion unit: the integer in
// the low word of 2^52 + 2^31, minus that
__device__ __forceinline__ double i32_to_f64(uint32_t v) {
  return __hiloint2double(0x43300000, (int)(v ^ 0x80000000u)) - 4503601774854144.0;
}

// C (m x n, column-major) -= A B from the digits, in two passes over K per
// tile: the sums s + t = 7, 6, 5, 4 (24 products), then 3, 2, 1, 0 (10
// products of the four leading digits), four 128-column accumulators each.
// Persistent over tiles_per_cta consecutive tiles (rows fastest, so neighbours
// in time share B):
//   warp 0 / lane 0   per 64-deep K block, one bulk copy of A's digits and one
//                     of B's (115 KB in the first pass, 66 KB in the second;
//                     the digits lie in global memory as the swizzled tiles
//                     the MMAs read) into a 2-stage ring;
//   warp 1 / lane 0   the pass's MMAs, accumulator by accumulator;
//   warps 2..9        L2 prefetch of the tile of C, then accumulator by
//                     accumulator as each is done: read (warp w: TMEM lanes 32
//                     (w % 4).., 64 columns), released to the next pass's
//                     MMAs, added to the FP64 sum in registers; after the
//                     second pass the update of C.
// A MMA of M = 128 takes 64 cycles for N = 64 and N = 128 alike (timed with
// the loads left out: 69 and 71), so one pass with eight 64-column
// accumulators ran at half the rate: 6144 x 6144 x 256 took 318 us of MMAs
// against 169. The loads alone take a quarter of that. Every wait is bounded,
// as in fp_tc.cu.
__global__ void __launch_bounds__(THREADS, 1)
k_i8_gemm_sub(const uint8_t* __restrict__ ad, const uint8_t* __restrict__ bd, int m, int n, int tiles_per_cta,
              const double* __restrict__ sa, const double* __restrict__ sb, double* __restrict__ C, int64_t ldc,
              int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
  uint64_t* empty = full + STAGES;
  uint64_t* accf = empty + STAGES;
  uint64_t* acce = accf + PG;
  uint64_t* drain = acce + PG;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = (m + BM - 1) / BM, ntiles = mt * ((n + BN - 1) / BN);
  const int t0 = blockIdx.x * tiles_per_cta, t1 = min(ntiles, t0 + tiles_per_cta);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int j = 0; j < PG; ++j) { mbar_init(&accf[j], 1); mbar_init(&acce[j], EPI_WARPS); }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(PG * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {   // producer
      int it = 0, issued = 0;
      for (int t = t0; t < t1 && !*(volatile int*)abort_flag; ++t) {
        const uint8_t* at = ad + (size_t)(t % mt) * NK * BLOCK;
        const uint8_t* bt = bd + (size_t)(t / mt) * NK * BLOCK;
        for (int q = 0; q < 2 * NK; ++q, ++it) {   // both passes' K blocks
          const int s = it % STAGES;
          const uint32_t bytes = q < NK ? BLOCK : PG * DIG;
          if (it >= STAGES && !mbar_wait(&empty[s], ((it / STAGES) - 1) & 1)) { *abort_flag = 1; break; }
          if (*(volatile int*)abort_flag) break;
          mbar_expect_tx(&full[s], 2 * bytes);
          bulk_load(smem + s * STAGE, at + (size_t)(q % NK) * BLOCK, bytes, &full[s]);
          bulk_load(smem + s * STAGE + BLOCK, bt + (size_t)(q % NK) * BLOCK, bytes, &full[s]);
          issued = it + 1;
        }
      }
      if (*(volatile int*)abort_flag)   // drain the copies this CTA issued before leaving
        for (int q = (issued > STAGES ? issued - STAGES : 0); q < issued; ++q)
          mbar_wait(&full[q % STAGES], (q / STAGES) & 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {   // MMA issuer
      int it = 0, u = 0;   // stages, passes
      bool ok = true;
      auto pass = [&](auto top) {   // the sums top .. top - PG + 1
        for (int kb = 0; ok && kb < NK; ++kb, ++it) {
          const int st = it % STAGES;
          if (!mbar_wait(&full[st], (it / STAGES) & 1)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t dA = sdesc64(smem_u32(smem + st * STAGE));
          const uint64_t dB = sdesc64(smem_u32(smem + st * STAGE + BLOCK));
#pragma unroll 1
          for (int kk = 0; ok && kk < KB / 32; ++kk) {
            const bool first = kb == 0 && kk == 0, last = kb == NK - 1 && kk == KB / 32 - 1;
            const uint64_t off = (uint64_t)(kk * 32 >> 4);
#pragma unroll
            for (int j = 0; j < PG; ++j) {
              constexpr int T = decltype(top)::value;
              const int g = T - j;
              if (first && u > 0 && ok) {
                ok = mbar_wait(&acce[j], (u - 1) & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              }
#pragma unroll
              for (int s = 0; s < S; ++s)
                if (g - s >= 0 && g - s < S)
                  umma_i8(tmem + (uint32_t)(j * BN), dA + off + (uint64_t)(s * DIG >> 4),
                          dB + off + (uint64_t)((g - s) * DIG >> 4), first && s == (g < S ? 0 : g - S + 1) ? 0u : 1u);
              if (last) umma_commit(&accf[j]);
            }
          }
          umma_commit(&empty[st]);
        }
        ++u;
      };
      for (int t = t0; ok && t < t1 && !*(volatile int*)abort_flag; ++t) {
        pass(std::integral_constant<int, G - 1>{});
        if (ok) pass(std::integral_constant<int, PG - 1>{});
      }
      if (!ok) *(volatile int*)abort_flag = 1;
      if (*(volatile int*)abort_flag && it > 0) {   // MMAs still in flight must finish before TMEM is freed
        umma_commit(drain);
        mbar_wait(drain, 0);
      }
    }
  } else {   // epilogue
    const int q = warp & 3, half = (warp - 2) >> 2;
    int u = 0;
    bool ok = true;
    for (int t = t0; ok && t < t1; ++t) {
      const int m0 = (t % mt) * BM, n0 = (t / mt) * BN + half * 64;
      const int r0 = m0 + q * 32, row = r0 + lane;
      const int nc = min(64, n - n0);
      // the warp's part of C: 64 columns of two 128-byte lines, on the load
      // path (bulk prefetches queue before the digits' copies)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cc = (lane >> 1) + 16 * i, rr = r0 + 16 * (lane & 1);
        if (cc < nc && rr < m) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (int64_t)(n0 + cc) * ldc + rr));
      }
      double acc[64];
#pragma unroll
      for (int e = 0; e < 64; ++e) acc[e] = 0.0;
#pragma unroll 1
      for (int p = 0; ok && p < 2; ++p, ++u)
#pragma unroll 1
        for (int j = 0; j < PG; ++j) {
          // warp-uniform: tcgen05.ld is a .sync.aligned warp instruction
          ok = __all_sync(0xffffffffu, mbar_wait(&accf[j], u & 1));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(j * BN + half * 64);
#pragma unroll
          for (int c16 = 0; c16 < 64; c16 += 16) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(base + (uint32_t)c16));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[c16 + e] = fma(acc[c16 + e], 0.00390625, i32_to_f64(v[e]));
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[j]);
        }
      if (!ok) {
        if (lane == 0) *(volatile int*)abort_flag = 1;
        break;
      }
      if (row < m) {
        const double s = sa[row];
        double* cp = C + (int64_t)n0 * ldc + row;
#pragma unroll
        for (int c8 = 0; c8 < 64; c8 += 8) {
          double old[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) old[e] = c8 + e < nc ? cp[(int64_t)(c8 + e) * ldc] : 0.0;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (c8 + e < nc) cp[(int64_t)(c8 + e) * ldc] = fma(-(acc[c8 + e] * s), __ldg(sb + n0 + c8 + e), old[e]);
        }
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && *(volatile int*)abort_flag) atomicOr(status, (int)DEV_TIMEOUT);
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PG * BN) : "memory");
}

// ---------------------------------------------------------------------------
// The digits. A lane holds 16 consecutive k of a row (of A) or column (of B),
// 16 lanes the whole of it; the largest |x| by its bit pattern, so that
// infinities and NaNs win and make the scale NaN: they reach every entry
// of that row or column of C, as in a product that meets them. They are stored
// as the MMAs' shared-memory tiles: blocks of 128 rows, per block and 64-deep K
// block the seven digits, each 128 rows of 64 bytes whose 16-byte pieces are
// permuted by the 64-byte swizzle (address bits 4-5 ^ bits 7-8).
__device__ __forceinline__ void digits16(const double (&x)[16], uint8_t* __restrict__ dig, int row, int kg,
                                         double* __restrict__ scale) {
  unsigned long long mx = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x[i]) & 0x7fffffffffffffffull;
    mx = b > mx ? b : mx;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = b > mx ? b : mx;
  }
  const int be = (int)(mx >> 52);          // biased exponent: |x| < 2^(be - 1022)
  const bool bad = be == 2047;
  // entries of a row that is all below 2^-900 keep the digits down to 2^-954
  const int ea = be < 123 ? -899 : be - 1022;
  const double up = bad ? 0.0 : __longlong_as_double((long long)(54 - ea + 1023) << 52);   // 2^(54 - ea)
  uint32_t w[S][4];
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) w[s][i] = 0u;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    // balanced digits of N = rint(x 2^(54 - ea)), |N| <= 2^54: the bytes of N + 0x80..80, less 128 each
    const unsigned long long b =
        ((unsigned long long)__double2ll_rn(x[i] * up) + 0x0080808080808080ull) ^ 0x0080808080808080ull;
#pragma unroll
    for (int s = 0; s < S; ++s) w[s][i / 4] |= (uint32_t)((b >> (8 * (S - 1 - s))) & 0xffu) << (8 * (i & 3));
  }
  const int r = row % BM;
  uint8_t* out = dig + ((size_t)(row / BM) * NK + kg / 4) * BLOCK + r * KB + (((kg & 3) ^ ((r >> 1) & 3)) << 4);
#pragma unroll
  for (int s = 0; s < S; ++s)
    *reinterpret_cast<uint4*>(out + s * DIG) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
  // the top digits' products carry 2^(96 - 108 + ea + eb): 2^-6 of it here, 2^-6 in the other operand
  if (scale) *scale = bad ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(1.0, ea - 6);
}

// rows of A (column-major, 256 columns): 32 rows a CTA through shared memory
constexpr int SPITCH = KP + KP / 16 + 1;   // doubles a row; k sits at k + k / 16 (no bank conflicts either way)
constexpr int SLICE_SMEM = 32 * SPITCH * 8;
__global__ void __launch_bounds__(512)
k_i8_rows(const double* __restrict__ A, int64_t lda, int m, uint8_t* __restrict__ dig, double* __restrict__ scale) {
  extern __shared__ double t[];
  const int r0 = blockIdx.x * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool in = r0 + lane < m;
#pragma unroll
  for (int i = 0; i < KP / 16; ++i) {
    const int k = w + 16 * i;
    t[lane * SPITCH + k + (k >> 4)] = in ? A[(int64_t)k * lda + r0 + lane] : 0.0;
  }
  __syncthreads();
  const int r = threadIdx.x >> 4, kg = threadIdx.x & 15;
  double x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = t[r * SPITCH + kg * 17 + i];
  // every lane takes part in the row's reduction; rows past the end write nothing of use (their digits are zero)
  digits16(x, dig, r0 + r, kg, kg == 0 && r0 + r < m ? scale + r0 + r : nullptr);
}

// columns of B (column-major, 256 rows)
__global__ void __launch_bounds__(256)
k_i8_cols(const double* __restrict__ B, int64_t ldb, int n, uint8_t* __restrict__ dig, double* __restrict__ scale) {
  const int j = blockIdx.x * 16 + (threadIdx.x >> 4), kg = threadIdx.x & 15;
  double x[16];
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const double2 v = j < n ? *reinterpret_cast<const double2*>(B + (int64_t)j * ldb + kg * 16 + i) : make_double2(0, 0);
    x[i] = v.x;
    x[i + 1] = v.y;
  }
  digits16(x, dig, j, kg, kg == 0 && j < n ? scale + j : nullptr);
}

}  // namespace i8

// Digit scratch of up to n rows of A and n columns of B, two sets (panel
// parity): per set A's digits, B's digits, then the scales of both; whole
// blocks of rows.
int i8_scratch(fp_ctx* c, int64_t n) {
  const int64_t np = round_up(n, i8::BM);
  if (c->i8_cap >= np) return FP_OK;
  for (int s = 0; s < 2; ++s) {
    if (c->d_i8[s]) cudaFree(c->d_i8[s]);
    c->d_i8[s] = nullptr;
  }
  c->i8_cap = 0;
  for (int s = 0; s < 2; ++s)
    FP_CUDA_TRY(c->err, cudaMalloc(&c->d_i8[s], (size_t)np * (2 * i8::S * i8::KP + 2 * sizeof(double))));
  c->i8_cap = np;
  return FP_OK;
}

namespace {
struct I8Set {
  uint8_t *a, *b;
  double *sa, *sb;
};
I8Set i8_set(fp_ctx* c, int set) {
  const size_t np = (size_t)c->i8_cap, dig = np * i8::S * i8::KP;
  uint8_t* p = c->d_i8[set];
  return {p, p + dig, reinterpret_cast<double*>(p + 2 * dig), reinterpret_cast<double*>(p + 2 * dig) + np};
}
}  // namespace

int i8_slice_rows(fp_ctx* c, int set, const double* A, int64_t lda, int64_t m) {
  static SmemAttr attr;
  FP_CUDA_TRY(c->err, attr.ensure(i8::k_i8_rows, i8::SLICE_SMEM));
  const I8Set s = i8_set(c, set);
  TraceScope tr(c, TR_SPLIT_A);
  i8::k_i8_rows<<<(unsigned)((m + 31) / 32), 512, i8::SLICE_SMEM, c->stream>>>(A, lda, (int)m, s.a, s.sa);
  ++c->nlaunch;
  FP_CUDA_TRY(c->err, cudaGetLastError());
  return FP_OK;
}

int i8_gemm_sub(fp_ctx* c, int set, const double* B, double* C, int64_t ld, int64_t m, int64_t col0, int64_t n) {
  if (m <= 0 || n <= 0) return FP_OK;
  const I8Set s = i8_set(c, set);
  uint8_t* bd = s.b + (size_t)col0 * i8::S * i8::KP;   // col0 is a multiple of the column blocks
  {
    TraceScope tr(c, TR_SPLIT_B);
    i8::k_i8_cols<<<(unsigned)((n + 15) / 16), 256, 0, c->stream>>>(B, ld, (int)n, bd, s.sb + col0);
    ++c->nlaunch;
    FP_CUDA_TRY(c->err, cudaGetLastError());
  }
  static SmemAttr attr;
  FP_CUDA_TRY(c->err, attr.ensure(i8::k_i8_gemm_sub, i8::SMEM));
  const int64_t tiles = ((m + i8::BM - 1) / i8::BM) * ((n + i8::BN - 1) / i8::BN);
  const int tpc = (int)std::max<int64_t>(1, std::min<int64_t>(8, tiles / (4 * num_sms())));
  const int ev = kt_begin(c);
  TraceScope tr(c, TR_GEMM_SIMT);
  i8::k_i8_gemm_sub<<<(unsigned)((tiles + tpc - 1) / tpc), i8::THREADS, i8::SMEM, c->stream>>>(
      s.a, bd, (int)m, (int)n, tpc, s.sa, s.sb + col0, C, ld, c->d_status);
  kt_end(c, ev, 2.0 * (double)m * (double)n * i8::KP, (double)m * (double)n);
  ++c->nlaunch;
  FP_CUDA_TRY(c->err, cudaGetLastError());
  return FP_OK;
}

}  // namespace fpb
