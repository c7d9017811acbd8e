// Complex128 products on the 8-bit integer tensor path (tcgen05 kind::i8).
//
//   C[e + ldc j] = alpha sum_k w[k % wmod] A[e + lda k] B[j + ldb k] + beta C[e + ldc j]
//
// the GEMM of the dense and separable-sum contractions
// (_production_static_contraction!, numerics/optimized/production_operators.jl:
// 402-465).  tcgen05 has no FP64 kind and the FP64 tensor path (mma.sync f64)
// stops at 37 TF/s, while kind::i8 measures 4.2 POP/s with exact int32 sums.
//
// Operands.  Every row of A (and of B) is scaled by a power of two so that its
// largest part lies in [2^60, 2^61), rounded to an integer (2^-61 of the row
// maximum) and written in 8 balanced base-256 digits x = sum_s d_s 256^(7-s),
// -128 <= d_s < 128; one 64-bit add and xor give all 8 digits.  The complex
// product takes three real ones, exact on the integers up to the digit
// products left out,
//   P0 = Re A Re B,  P1 = Im A Im B,  P2 = (Re A + Im A)(Re B + Im B),
//   Re C = P0 - P1,  Im C = P2 - P0 - P1,
// each the digit products with s + t <= 7: 36 of 64 int8 GEMMs.  What is left
// out lies under 2^-64 of a product of row maxima.  On the kernels and Green
// functions of an SCBA (row rms 0.05 to 0.2 of the row maximum) the error
// against 64-bit arithmetic with exact sums is 1e-16 of the result, against
// 5e-16 to 1.5e-15 for FP64 accumulation at K = 216 to 640, which grows with
// K.  A row with a non-finite value gives NaN in its row (column) of C.
//
// Sums.  The digit products of one diagonal s + t share an int32 accumulator:
// at most 8 of them at s + t = 7, so K <= 16320 per accumulation keeps
// 8 * K * 2^14 below 2^31; a longer K takes several.  Four diagonals of a
// 128 x BN tile (BN <= 128) fill the 512 columns of tensor memory: two passes
// over K per product, diagonals 4..7 (26 MMAs per 32 of K) and 0..3 (10).
// The four sums are combined exactly in 64 bits, converted once and added to
// C in FP64.
//
// Kernel: persistent CTAs (one per SM) of 320 threads walk the tiles.  Warp 8
// streams operand blocks with untiled bulk copies into a 3-stage ring (the
// split kernels write the operands in the order the MMA reads them: 16-byte
// K chunks of consecutive rows), warp 9 issues the MMAs, warps 0-7 add the
// sums to C.  A stage holds 8 digit tiles of A and B: one 32-wide block of K
// with all 8 digits, or two with the 4 leading ones.
//
// Bound: the int8 rate and the power limit (980 of 1000 W drawn).  2048 x 8192
// x 8192 (both Keldysh components of an operator with 32 momenta and 16
// states): 9.9 ms = 3.0 POP/s of the 4.2 POP/s that resident operands reach,
// plus 1.2 ms for the split; the FP64 tensor path takes 36 ms.
#include <algorithm>
#include <climits>

#include "kernels.cuh"
#include "tc_prims.cuh"

namespace qcl {

constexpr int I8_BM = 128, I8_MAXBN = 128, I8_KB = 32, I8_S = 8;
constexpr int I8_STAGES = 3, I8_DRAIN = 8, I8_THREADS = 32 * (I8_DRAIN + 2);
constexpr int I8_A_TILE = I8_BM * I8_KB;            // bytes of one digit tile of A
constexpr int I8_SEG_KB = 16320 / I8_KB;            // K blocks per accumulation (even)
constexpr int I8_TOP = 61;                          // |x| < 2^61
constexpr int I8_BAD = 1 << 20;                     // exponent of a row with a non-finite value
static_assert(8ll * I8_SEG_KB * I8_KB * 128 * 128 < (1ll << 31), "int32 accumulation");

__device__ long long g_i8_main_wait_limit = TC_WAIT_LIMIT;

template <int BN> struct I8Shape {
  static constexpr int B_TILE = BN * I8_KB;
  static constexpr int SUB = I8_A_TILE + B_TILE;     // one digit tile of A and of B
  static constexpr int STAGE = 8 * SUB;
  static constexpr int SMEM = I8_STAGES * STAGE + 1024 + 128;
};

// K-major operand without swizzle: 8-row x 16-byte cores, 128 B apart along
// the rows, `rows` * 16 B apart along K.
__device__ __forceinline__ uint64_t i8_desc(uint32_t saddr, int rows) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)rows << 16) | ((uint64_t)8 << 32) | ((uint64_t)1 << 46);
}
// D s32, A/B s8, both K-major.
template <int BN> __device__ __forceinline__ constexpr uint32_t i8_idesc() {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(I8_BM >> 4) << 24);
}
__device__ __forceinline__ void i8_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0)
      : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

struct I8Args {
  const signed char *A, *B;      // [plane][K block][digit][K half][row][16]
  long long a_plane, b_plane;    // bytes per plane (Re, Im, Re + Im)
  int a_rows, b_rows;            // padded rows
  int nkb;                       // K blocks (even)
  int mtiles, ntiles;            // tiles of C
  int M, mpad;                   // rows of C per field, padded rows per field
  int N;                         // columns of C
  const int *ea, *eb;            // row exponents
  Cx<double>* C[2];              // output fields: rows [f mpad, f mpad + M)
  long long ldc;
  double alpha, beta;
  int* status;
};

// The digit products of a stage.  PASS 0 (diagonals 4..7, one K block): as
// digits arrive in the order 0 7 1 6 2 5 3 4; PASS 1 (diagonals 0..3).
// Accumulator i holds diagonal 4 + i or i.
template <int BN, int PASS>
__device__ __forceinline__ void i8_issue(uint32_t st, uint32_t tmem, bool first) {
  using S = I8Shape<BN>;
  constexpr uint32_t idesc = i8_idesc<BN>();
  const uint64_t a0 = i8_desc(st, I8_BM), b0 = i8_desc(st + I8_A_TILE, BN);
  constexpr int BLOCKS = PASS == 0 ? 1 : 2, ND = PASS == 0 ? 8 : 4;
#pragma unroll
  for (int kb = 0; kb < BLOCKS; ++kb)
#pragma unroll
    for (int s = 0; s < ND; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = PASS == 0 ? 4 + i : i, t = d - s;
        if (t < 0 || t >= ND) continue;
        const uint32_t oa = (uint32_t)((kb * ND + s) * S::SUB) >> 4, ob = (uint32_t)((kb * ND + t) * S::SUB) >> 4;
        i8_mma(tmem + i * 128, a0 + oa, b0 + ob, idesc, (kb == 0 && s == 0) ? (first ? 0u : 1u) : 1u);
      }
}

template <int BN> __global__ void __launch_bounds__(I8_THREADS, 1) i8_gemm_kernel(const __grid_constant__ I8Args p) {
  using S = I8Shape<BN>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - raw);
  const uint32_t bars = base + I8_STAGES * S::STAGE;
  const uint32_t full = bars, empty = bars + 8 * I8_STAGES, acc_full = bars + 16 * I8_STAGES, acc_empty = acc_full + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + I8_STAGES * S::STAGE + 16 * I8_STAGES + 16);
  __shared__ volatile int s_fail;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = p.mtiles * p.ntiles;
  const int ntile = (int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int nseg = (p.nkb + I8_SEG_KB - 1) / I8_SEG_KB;
  const long long lim = g_i8_main_wait_limit;
  if (threadIdx.x == 0) {
    for (int i = 0; i < I8_STAGES; ++i) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 32 * I8_DRAIN);
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == I8_DRAIN + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Every role walks the same units: tile, K segment, product (plane), pass.
  // `it` counts stages over the CTA's units (ring position and phase), `u` units.
  int it = 0, u = 0;
  int loaded = 0, issued = 0;

  if (warp == I8_DRAIN) {
    // ---- producer: lane i copies piece i of a stage (8 digit tiles x A/B x K half) ----
    const int sub = lane >> 2, isb = (lane >> 1) & 1, kc = lane & 1;
    const uint32_t dst = (uint32_t)(sub * S::SUB + (isb ? I8_A_TILE + kc * BN * 16 : kc * I8_BM * 16));
    const uint32_t bytes = isb ? BN * 16 : I8_BM * 16;
    const long long rows = isb ? p.b_rows : p.a_rows;
    bool ok = true;
    for (int i = 0; i < ntile && ok; ++i) {
      const int t = (int)blockIdx.x + i * (int)gridDim.x;
      const long long row0 = isb ? (long long)(t / p.mtiles) * BN : (long long)(t % p.mtiles) * I8_BM;
      for (int seg = 0; seg < nseg && ok; ++seg)
        for (int pl = 0; pl < 3 && ok; ++pl) {
          const signed char* plane = isb ? p.B + pl * p.b_plane : p.A + pl * p.a_plane;
          const int k0 = seg * I8_SEG_KB, k1 = min(p.nkb, k0 + I8_SEG_KB);
          for (int pass = 0; pass < 2 && ok; ++pass)
            for (int kb = k0; kb < k1; kb += pass ? 2 : 1, ++it) {
              const int s = it % I8_STAGES;
              if (it >= I8_STAGES && !mbar_wait(empty + 8 * s, (uint32_t)((it / I8_STAGES - 1) & 1), lim)) s_fail = 1;
              if (__any_sync(0xffffffffu, s_fail != 0)) {
                ok = false;
                break;
              }
              const int kk = pass ? kb + (sub >> 2) : kb, dg = pass ? sub & 3 : sub;
              if (lane == 0) mbar_expect_tx(full + 8 * s, S::STAGE);
              __syncwarp();
              bulk_load(base + s * S::STAGE + dst, plane + ((((long long)kk * I8_S + dg) * 2 + kc) * rows + row0) * 16,
                        bytes, full + 8 * s);
              loaded = it + 1;
            }
        }
    }
  } else if (warp == I8_DRAIN + 1) {
    // ---- MMA issue ----
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < ntile && ok; ++i)
        for (int seg = 0; seg < nseg && ok; ++seg)
          for (int pl = 0; pl < 3 && ok; ++pl) {
            const int k0 = seg * I8_SEG_KB, k1 = min(p.nkb, k0 + I8_SEG_KB);
            for (int pass = 0; pass < 2 && ok; ++pass, ++u) {
              if (u > 0 && !mbar_wait(acc_empty, (uint32_t)((u - 1) & 1), lim)) ok = false;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              for (int kb = k0; ok && kb < k1; kb += pass ? 2 : 1, ++it) {
                const int s = it % I8_STAGES;
                if (s_fail || !mbar_wait(full + 8 * s, (uint32_t)((it / I8_STAGES) & 1), lim)) {
                  ok = false;
                  break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (pass == 0) i8_issue<BN, 0>(base + s * S::STAGE, tmem, kb == k0);
                else i8_issue<BN, 1>(base + s * S::STAGE, tmem, kb == k0);
                tc_commit(empty + 8 * s);
                issued = it + 1;
              }
              if (ok) tc_commit(acc_full);
            }
          }
      if (!ok) s_fail = 1;
      // the tensor memory is released below: let every issued MMA finish (bounded)
      if (issued > 0) mbar_wait(empty + 8 * ((issued - 1) % I8_STAGES), (uint32_t)(((issued - 1) / I8_STAGES) & 1));
    }
  } else {
    // ---- sums into C ----
    const uint32_t tlane = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int CH = BN / 2;  // columns per warp
    const int c0 = (warp >> 2) * CH;
    bool ok = true;
    for (int i = 0; i < ntile && ok; ++i) {
      const int t = (int)blockIdx.x + i * (int)gridDim.x;
      const int r = (t % p.mtiles) * I8_BM + (warp & 3) * 32 + lane;
      const int f = r / p.mpad, e = r - f * p.mpad;
      const int n0 = (t / p.mtiles) * BN + c0;
      const bool row_ok = e < p.M;
      const int ea = p.ea[r];
      Cx<double>* C = (f ? p.C[1] : p.C[0]) + (row_ok ? e : 0);
      for (int seg = 0; seg < nseg && ok; ++seg)
        for (int pl = 0; pl < 3 && ok; ++pl)
          for (int pass = 0; pass < 2; ++pass, ++u) {
            const bool stop = __any_sync(0xffffffffu, s_fail != 0);
            if (!__all_sync(0xffffffffu, !stop && mbar_wait(acc_full, (uint32_t)(u & 1), lim))) {
              ok = false;
              s_fail = 1;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool first = seg == 0 && pl == 0 && pass == 0;
            // x = X 2^(e - 61); the four sums in units of 256^7 (pass 0) or 256^11
            const int unit = ea - 2 * I8_TOP + (pass ? 88 : 56);
            const double sre = pl == 0 ? p.alpha : pl == 1 ? -p.alpha : 0.0, sim = pl == 2 ? p.alpha : -p.alpha;
#pragma unroll 1
            for (int c = 0; c < CH; c += 8) {
              int v[4][8];
#pragma unroll
              for (int q = 0; q < 4; ++q) tmem_ld8(tmem + tlane + (uint32_t)(q * 128 + c0 + c), v[q]);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              Cx<double> o[8];
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                o[q] = cx<double>(0, 0);
                if (row_ok && n0 + c + q < p.N && (!first || p.beta != 0.0)) o[q] = C[p.ldc * (n0 + c + q)];
              }
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                if (!row_ok || n0 + c + q >= p.N) continue;
                const long long x =
                    ((((long long)v[0][q] << 8) + v[1][q]) * 65536) + (((long long)v[2][q] << 8) + v[3][q]);
                const int ex = unit + p.eb[n0 + c + q];
                double y = scalbn((double)x, ex);
                if (ex >= I8_BAD / 2) y = NAN;
                if (first) o[q] = p.beta == 0.0 ? cx<double>(0, 0) : p.beta * o[q];
                o[q].x = fma(sre, y, o[q].x);
                o[q].y = fma(sim, y, o[q].y);
                C[p.ldc * (n0 + c + q)] = o[q];
              }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(acc_empty);
          }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) record_status(p.status, QCL_TIMEOUT, (long long)blockIdx.x);
  if (warp == I8_DRAIN + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  // after a failure copies may still be in flight into this CTA's shared memory
  if (warp == I8_DRAIN && lane == 0 && s_fail)
    for (int kl = loaded > I8_STAGES ? loaded - I8_STAGES : 0; kl < loaded; ++kl)
      mbar_wait(full + 8 * (kl % I8_STAGES), (uint32_t)((kl / I8_STAGES) & 1));
}

// ---------------------------------------------------------------------------
// Operand preparation.  Row r of the operand is element (r % rpad) of field
// r / rpad: X[f][e + ld k] w[k % wmod], e < rows, k < K; zero elsewhere.
// ---------------------------------------------------------------------------
struct I8Src {
  const Cx<double>* X[2];
  long long ld;
  const double* w;
  int wmod;
  int rows, rpad, total;  // rows per field, padded rows per field, rows of the operand
  int K;
};

// Largest part of each row as FP64 bits (non-negative values order as
// integers; a non-finite value gives +inf), which the caller zeroes first.
__global__ void i8_row_max_kernel(I8Src a, unsigned long long* __restrict__ rowmax, int kper) {
  __shared__ double red[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + tx, f = r / a.rpad, e = r - f * a.rpad;
  const int k0 = blockIdx.y * kper, k1 = min(a.K, k0 + kper);
  double mx = 0.0;
  if (e < a.rows) {
    const Cx<double>* X = (f ? a.X[1] : a.X[0]) + e;
#pragma unroll 4
    for (int k = k0 + ty; k < k1; k += 8) {
      const double w = a.w ? a.w[k % a.wmod] : 1.0;
      const Cx<double> v = X[a.ld * k];
      const double x = fabs(v.x * w), y = fabs(v.y * w);
      mx = (isfinite(x) && isfinite(y)) ? fmax(mx, fmax(x, y)) : INFINITY;
    }
  }
  red[ty][tx] = mx;
  __syncthreads();
  if (ty == 0 && e < a.rows) {
    for (int q = 1; q < 8; ++q) mx = fmax(mx, red[q][tx]);
    atomicMax(rowmax + r, (unsigned long long)__double_as_longlong(mx));
  }
}

// 4 x 4 byte transpose: out[i] = byte i of each of a, b, c, d.
__device__ __forceinline__ void byte_transpose(unsigned a, unsigned b, unsigned c, unsigned d, unsigned (&out)[4]) {
  const unsigned ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
  const unsigned cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
  out[0] = __byte_perm(ab0, cd0, 0x5410);
  out[1] = __byte_perm(ab0, cd0, 0x7632);
  out[2] = __byte_perm(ab1, cd1, 0x5410);
  out[3] = __byte_perm(ab1, cd1, 0x7632);
}

// One thread per row and 16-wide K half: 16 values, their 3 x 16 integers, and
// 3 x 8 digit rows of 16 bytes.  A warp reads and writes 512 contiguous bytes.
__global__ void __launch_bounds__(256) i8_split_kernel(I8Src a, const unsigned long long* __restrict__ rowmax,
                                                       int* __restrict__ exps, signed char* __restrict__ out,
                                                       long long plane, int halves) {
  const int r = blockIdx.x * 32 + (threadIdx.x & 31), f = r / a.rpad, e = r - f * a.rpad;
  const int half = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (half >= halves) return;
  const bool live = e < a.rows;
  const double mx = live ? __longlong_as_double((long long)rowmax[r]) : 0.0;
  int ex = 0;
  const bool bad = isinf(mx);
  if (mx > 0.0 && !bad) frexp(mx, &ex);
  if (half == 0) exps[r] = bad ? I8_BAD : ex;
  // x 2^(61 - ex) in two exact steps (either factor alone stays in range)
  const int sh = I8_TOP - ex, sh1 = sh / 2;
  const double s1 = ldexp(1.0, sh1), s2 = ldexp(1.0, sh - sh1);
  const bool use = live && !bad;
  const Cx<double>* X = (f ? a.X[1] : a.X[0]) + e;
  long long xr[16], xi[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int k = half * 16 + i;
    Cx<double> v = cx<double>(0, 0);
    if (use && k < a.K) {
      v = X[a.ld * k];
      const double w = a.w ? a.w[k % a.wmod] : 1.0;
      v = cx<double>(v.x * w, v.y * w);
    }
    xr[i] = __double2ll_rn(v.x * s1 * s2);
    xi[i] = __double2ll_rn(v.y * s1 * s2);
  }
  signed char* dst = out + ((long long)(half >> 1) * I8_S * 2 + (half & 1)) * (long long)a.total * 16 + (long long)r * 16;
  const long long dstep = 2ll * a.total * 16;  // next digit
  constexpr unsigned long long BIAS = 0x8080808080808080ull;
#pragma unroll
  for (int pl = 0; pl < 3; ++pl) {
    unsigned lo[8][4];  // digit (0 = least significant) x 4 words of 4 K values
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      unsigned l[4], h[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = 4 * g + q;
        const long long x = pl == 0 ? xr[i] : pl == 1 ? xi[i] : xr[i] + xi[i];
        const unsigned long long z = ((unsigned long long)x + BIAS) ^ BIAS;
        l[q] = (unsigned)z;
        h[q] = (unsigned)(z >> 32);
      }
      unsigned t[4];
      byte_transpose(l[0], l[1], l[2], l[3], t);
#pragma unroll
      for (int q = 0; q < 4; ++q) lo[q][g] = t[q];
      byte_transpose(h[0], h[1], h[2], h[3], t);
#pragma unroll
      for (int q = 0; q < 4; ++q) lo[4 + q][g] = t[q];
    }
#pragma unroll
    for (int s = 0; s < I8_S; ++s)
      *reinterpret_cast<uint4*>(dst + pl * plane + s * dstep) =
          make_uint4(lo[7 - s][0], lo[7 - s][1], lo[7 - s][2], lo[7 - s][3]);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

static int sm_count() {
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Clocks of one MMA (M = 128, K = 32) by tile width, measured.
static double i8_clk(int bn) { return bn == 128 ? 71 : bn == 112 ? 64 : bn == 96 ? 58 : 52; }

// Tile width whose waves over the SMs take the least time.
static int i8_pick_bn(int mtiles, int N, int sms, double* cost = nullptr) {
  int best = 128;
  double bc = -1;
  for (int bn : {128, 112, 96, 64}) {
    const double c = ceil_div((long long)mtiles * ceil_div(N, bn), sms) * i8_clk(bn);
    if (bc < 0 || c < 0.99 * bc) {
      bc = c;
      best = bn;
    }
  }
  if (cost) *cost = bc;
  return best;
}

struct I8Dims {
  int mpad, nkb;
  size_t a_row, b_row;  // bytes per operand row (digits, row maximum, exponent)
};
static I8Dims i8_dims(int M, int K) {
  I8Dims d;
  d.mpad = ceil_div(M, I8_BM) * I8_BM;
  d.nkb = ceil_div(K, 2 * I8_KB) * 2;
  d.a_row = d.b_row = 3 * (size_t)d.nkb * I8_KB * I8_S + 16;
  return d;
}
// Rows of a padded B panel: whole tiles of every width.
static int i8_bpad(int N) { return ceil_div(N, I8_MAXBN) * I8_MAXBN + I8_MAXBN; }

size_t i8_work_bytes(int M, int fields, int N, int K) {
  const I8Dims d = i8_dims(M, K);
  return (size_t)fields * d.mpad * d.a_row + (size_t)i8_bpad(N) * d.b_row + 4096;
}

// Whether the product is large enough for the split to pay (FP64 tensor path
// against this one, both passes and the split included):
//   rows x K x columns  2048 x 576^2: 192 / 181 us, 1000 x 1152^2: 374 / 279 us,
//   383 x 2048^2: 667 / 470 us, 1024 x 2048^2: 1301 / 530 us, 1024 x 8192^2:
//   17.98 / 6.92 ms; below the line 400 x 1152^2: 225 / 276 us, 128 x 2048^2:
//   392 / 462 us, 64 x 4096^2: 780 / 980 us (few row tiles, split costs remain).
bool i8_worthwhile(int M, int fields, int N, int K) {
  return (double)M * fields * N * K >= 1e9 && (long long)M * fields >= 192 && N >= 64 && K >= 64;
}

template <int BN> static int launch_i8_t(const I8Args& a, int sms, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(i8_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, I8Shape<BN>::SMEM));
    configured = true;
  }
  const int tiles = a.mtiles * a.ntiles;
  i8_gemm_kernel<BN><<<std::min(tiles, sms), I8_THREADS, I8Shape<BN>::SMEM, st>>>(a);
  QCL_LAUNCH_CHECK("i8_gemm_kernel");
  return QCL_OK;
}

static int i8_split(const I8Src& a, unsigned long long* rowmax, int* exps, signed char* out, int nkb, cudaStream_t st) {
  QCL_CUDA_CHECK(cudaMemsetAsync(rowmax, 0, (size_t)a.total * sizeof(unsigned long long), st));
  const int rb = a.total / 32;
  int ks = std::max(1, std::min(ceil_div(a.K, 64), 8 * 148 / rb));
  const int kper = ceil_div(a.K, ks);
  i8_row_max_kernel<<<dim3(rb, ceil_div(a.K, kper)), 256, 0, st>>>(a, rowmax, kper);
  QCL_LAUNCH_CHECK("i8_row_max_kernel");
  const long long plane = (long long)nkb * I8_S * 2 * a.total * 16;
  i8_split_kernel<<<dim3(rb, ceil_div(2 * nkb, 8)), 256, 0, st>>>(a, rowmax, exps, out, plane, 2 * nkb);
  QCL_LAUNCH_CHECK("i8_split_kernel");
  return QCL_OK;
}

int launch_i8_gemm(int M, int fields, int N, int K, const void* const* A, long long lda, const double* w, int wmod,
                   const void* B, long long ldb, void* const* C, long long ldc, double alpha, double beta, void* work,
                   size_t work_bytes, int* status, cudaStream_t st) {
  const I8Dims d = i8_dims(M, K);
  const int sms = sm_count();
  // panels: rows of A (one field) and columns of B that the work area holds
  int mp = 1, np = 1;
  auto panel = [](int n, int parts, int unit) { return std::min(n, ceil_div(ceil_div(n, parts), unit) * unit); };
  auto need = [&]() {
    const int m = panel(M, mp, I8_BM), n = panel(N, np, I8_MAXBN);
    return i8_work_bytes(m, fields, n, K);
  };
  while (need() > work_bytes) {
    const size_t ab = (size_t)fields * panel(M, mp, I8_BM) * d.a_row, bb = (size_t)panel(N, np, I8_MAXBN) * d.b_row;
    if (ab >= bb && panel(M, mp, I8_BM) > I8_BM) ++mp;
    else if (panel(N, np, I8_MAXBN) > I8_MAXBN) ++np;
    else if (panel(M, mp, I8_BM) > I8_BM) ++mp;
    else {
      set_last_error("i8 product: work area of %zu bytes is too small", work_bytes);
      return QCL_UNSUPPORTED;
    }
  }
  const int mpan = panel(M, mp, I8_BM), npan = panel(N, np, I8_MAXBN);
  for (int n0 = 0; n0 < N; n0 += npan) {
    const int n = std::min(npan, N - n0), bpad = i8_bpad(n);
    char* q = (char*)work;
    auto take = [&](size_t bytes) {
      char* r = q;
      q += (bytes + 255) / 256 * 256;
      return r;
    };
    unsigned long long* bmax = (unsigned long long*)take((size_t)bpad * 8);
    int* eb = (int*)take((size_t)bpad * 4);
    signed char* Bd = (signed char*)take(3 * (size_t)d.nkb * I8_KB * I8_S * bpad);
    int s;
    I8Src bs{{(const Cx<double>*)B + n0, nullptr}, ldb, nullptr, 1, n, bpad, bpad, K};
    if ((s = i8_split(bs, bmax, eb, Bd, d.nkb, st))) return s;
    for (int m0 = 0; m0 < M; m0 += mpan) {
      const int m = std::min(mpan, M - m0), mpad = ceil_div(m, I8_BM) * I8_BM, rows = fields * mpad;
      char* keep = q;
      unsigned long long* amax = (unsigned long long*)take((size_t)rows * 8);
      int* ea = (int*)take((size_t)rows * 4);
      signed char* Ad = (signed char*)take(3 * (size_t)d.nkb * I8_KB * I8_S * rows);
      q = keep;
      I8Src as{{(const Cx<double>*)A[0] + m0, fields > 1 ? (const Cx<double>*)A[1] + m0 : nullptr}, lda, w, wmod, m, mpad,
               rows, K};
      if ((s = i8_split(as, amax, ea, Ad, d.nkb, st))) return s;
      I8Args g{};
      g.A = Ad;
      g.B = Bd;
      g.a_plane = (long long)d.nkb * I8_S * 2 * rows * 16;
      g.b_plane = (long long)d.nkb * I8_S * 2 * bpad * 16;
      g.a_rows = rows;
      g.b_rows = bpad;
      g.nkb = d.nkb;
      g.mtiles = rows / I8_BM;
      g.M = m;
      g.mpad = mpad;
      g.N = n;
      g.ea = ea;
      g.eb = eb;
      for (int f = 0; f < fields; ++f) g.C[f] = (Cx<double>*)C[f] + m0 + ldc * n0;
      g.ldc = ldc;
      g.alpha = alpha;
      g.beta = beta;
      g.status = status;
      const int bn = i8_pick_bn(g.mtiles, n, sms);
      g.ntiles = ceil_div(n, bn);
      if (bn == 128) s = launch_i8_t<128>(g, sms, st);
      else if (bn == 112) s = launch_i8_t<112>(g, sms, st);
      else if (bn == 96) s = launch_i8_t<96>(g, sms, st);
      else s = launch_i8_t<64>(g, sms, st);
      if (s) return s;
    }
  }
  return QCL_OK;
}

int i8_set_wait_limit(long long rounds) {
  const long long v = rounds >= 0 ? rounds : TC_WAIT_LIMIT;
  QCL_CUDA_CHECK(cudaMemcpyToSymbol(g_i8_main_wait_limit, &v, sizeof(v)));
  return QCL_OK;
}

}  // namespace qcl
