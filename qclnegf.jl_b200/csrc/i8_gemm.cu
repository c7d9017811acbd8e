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
// each the digit products with s + t <= 7 (36 of 64 int8 GEMMs) or, where the
// accuracy asks for it, s + t <= 8 (43).  The family of methods is that of
// Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 2012).
//
// Accuracy.  Let MA and MB be the powers of two above the largest parts of the
// two rows.  The 7 digit products of the first diagonal left out are at most
// 2^14 each, in units of 2^(48-122): per term of K the error of one part of C
// is at most 3 x 2^-57.2 = 2^-55.6 of MA MB (three products in Im C) and, the
// digits being spread over their range, 2^-59.4 rms (1.2e-18 measured), which
// adds up as sqrt(K).  This is relative to the rows' maxima; an FP64 sum's error
// is relative to sum_k |a_k| |b_k|: 2K x 2^-53 of it at most, 0.6 to 29e-16 rms
// measured (least where few terms dominate).  So what decides is
//   S = sum_k |a_k| |b_k| / (MA MB):
// by the bounds the two meet at S = 0.08, by the rms at S = 1.2e-18 sqrt(K) /
// 1.2e-16 = sqrt(K) / 100.  The path runs only where every output lies above
// that: before it, the leading 7 bits of all entries (rounded down, so that
// their sum is a lower bound of S) go through one int8 product, 1/108 of the
// work.  One output below the line adds the diagonal s + t = 8 to the product;
// what is left then is the rounding of the operands, 2^-62 of the maxima per
// entry (2^-62.8 rms): S = 0.006 by the bounds, sqrt(K) / 1500 by the rms.  One
// output below that line rejects the product, which then takes the FP64 tensor
// path.  Outputs of a zero row are
// exact and exempt; a non-finite entry rejects.  Errors in units of sum |a| |b|,
// here / FP64 path:
//   normal entries, K = 1024 ... 8192: 3.4 ... 1.3e-18 / 6e-17
//   random form factors with SCBA fields, K = 8192 (S >= 1.5): 1.1e-17 / 5e-16
//   entries of one sign, K = 1024 ... 8192: 4e-17 / 9 ... 29e-16
// The screened kernels of a real stack, whose far couplings meet small entries
// only, go down to S = 1e-8 and are rejected.
//
// Sums.  The digit products of one diagonal s + t share an int32 accumulator:
// at most 8 of them, so K <= 16320 per accumulation keeps 8 * K * 2^14 below
// 2^31; a longer K takes several.  Four diagonals of a 128 x BN tile (BN <= 128)
// fill the 512 columns of tensor memory, so a product takes passes over K:
// diagonals 4..7 (26 MMAs per 32 of K) and 0..3 (10), or 5..8 (28), 1..4 (14)
// and 0 (1).  The sums of a pass are combined exactly in 64 bits, converted once
// and added to C in FP64.
//
// Kernel: persistent CTAs (one per SM) of 320 threads walk the tiles.  Warp 8
// streams operand blocks with untiled bulk copies into a 3-stage ring (the
// split kernels write the operands in the order the MMA reads them: 16-byte
// K chunks of consecutive rows), warp 9 issues the MMAs, warps 0-7 add the
// sums to C.  A stage holds up to 8 digit tiles of A and B: one 32-wide block of
// K with all 8 digits, two with the 4 leading ones, eight with one.
//
// Bound: the int8 rate and the power limit (980 of 1000 W drawn).  2048 x 8192
// x 8192 (both Keldysh components of an operator with 32 momenta and 16
// states): 9.9 ms = 3.0 POP/s of the 4.2 POP/s that resident operands reach,
// plus 1.2 ms for the split and 0.35 ms for the bound; the FP64 tensor path takes
// 36 ms.  With the extra diagonal about 12.5 ms.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"
#include "tc_prims.cuh"

namespace qcl {

constexpr int I8_BM = 128, I8_MAXBN = 128, I8_KB = 32, I8_S = 8;
constexpr int I8_STAGES = 3, I8_DRAIN = 8, I8_THREADS = 32 * (I8_DRAIN + 2);
constexpr int I8_A_TILE = I8_BM * I8_KB;            // bytes of one digit tile of A
constexpr int I8_SEG_KB = 16320 / I8_KB;            // K blocks per accumulation (even)
constexpr int I8_TOP = 61;                          // |x| < 2^61
constexpr int I8_BOUND_MAX_KB = 4096;               // further ones are left out of the bound (int32: 2^17 x 127^2 < 2^31)
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
  const unsigned long long *amax, *bmax;  // row maxima (FP64 bits)
  int* level;                    // of the product: I8_PLAIN, I8_WIDE or kI8Rejected
  int wide_line, reject_line;    // least sums of leading bits of the first two
  Cx<double>* C[2];              // output fields: rows [f mpad, f mpad + M)
  long long ldc;
  double alpha, beta;
  int* status;
};

// What a launch computes, and its passes over K: blocks of K and digits per
// stage, the lowest diagonal and the number of diagonals.
enum { I8_PLAIN = 0, I8_WIDE = 1, I8_BOUND = 3 };
static_assert(I8_PLAIN < I8_WIDE && I8_WIDE < kI8Rejected, "levels rise");
template <int MODE> struct I8Passes;
template <> struct I8Passes<I8_PLAIN> {
  static constexpr int PLANES = 3, PASSES = 2, SEG_KB = I8_SEG_KB;
  __device__ static constexpr int blocks(int pass) { return pass ? 2 : 1; }
  __device__ static constexpr int digits(int pass) { return pass ? 4 : 8; }
  __device__ static constexpr int low(int pass) { return pass ? 0 : 4; }
  __device__ static constexpr int sums(int) { return 4; }
};
template <> struct I8Passes<I8_WIDE> {
  static constexpr int PLANES = 3, PASSES = 3, SEG_KB = I8_SEG_KB;
  __device__ static constexpr int blocks(int pass) { return pass == 2 ? 8 : 1; }
  __device__ static constexpr int digits(int pass) { return pass == 0 ? 8 : pass == 1 ? 5 : 1; }
  __device__ static constexpr int low(int pass) { return pass == 0 ? 5 : pass == 1 ? 1 : 0; }
  __device__ static constexpr int sums(int pass) { return pass == 2 ? 1 : 4; }
};
template <> struct I8Passes<I8_BOUND> {  // the leading bits: one plane, one digit
  static constexpr int PLANES = 1, PASSES = 1, SEG_KB = I8_BOUND_MAX_KB;
  __device__ static constexpr int blocks(int) { return 8; }
  __device__ static constexpr int digits(int) { return 1; }
  __device__ static constexpr int low(int) { return 0; }
  __device__ static constexpr int sums(int) { return 1; }
};

// The digit products of a stage with `blocks` K blocks; as digits arrive in the
// order 0 7 1 6 2 5 3 4.  Accumulator i holds diagonal low + i; `first`: its
// sums start here.
template <int BN, int MODE, int PASS>
__device__ __forceinline__ void i8_issue(uint32_t st, uint32_t tmem, bool first, int blocks) {
  using S = I8Shape<BN>;
  using P = I8Passes<MODE>;
  constexpr int BLOCKS = P::blocks(PASS), ND = P::digits(PASS), LOW = P::low(PASS), SUMS = P::sums(PASS);
  constexpr uint32_t idesc = i8_idesc<BN>();
  static_assert(BLOCKS * ND <= 8, "stage");
  const uint64_t a0 = i8_desc(st, I8_BM), b0 = i8_desc(st + I8_A_TILE, BN);
#pragma unroll
  for (int kb = 0; kb < BLOCKS; ++kb) {
    if (kb >= blocks) break;
#pragma unroll
    for (int s = 0; s < ND; ++s)
#pragma unroll
      for (int i = 0; i < SUMS; ++i) {
        const int t = LOW + i - s;
        if (t < 0 || t >= ND) continue;
        const uint32_t oa = (uint32_t)((kb * ND + s) * S::SUB) >> 4, ob = (uint32_t)((kb * ND + t) * S::SUB) >> 4;
        const bool start = kb == 0 && (s == 0 || t == ND - 1);  // the diagonal's first product
        i8_mma(tmem + i * 128, a0 + oa, b0 + ob, idesc, start && first ? 0u : 1u);
      }
  }
}

// MODE I8_BOUND: raises *level where an output of two non-zero rows lies below
// a line.  I8_PLAIN, I8_WIDE: the product, if it has that level.
template <int BN, int MODE>
__global__ void __launch_bounds__(I8_THREADS, 1) i8_gemm_kernel(const __grid_constant__ I8Args p) {
  using S = I8Shape<BN>;
  using P = I8Passes<MODE>;
  {  // (one answer for the CTA: another one of the launch may raise it)
    const int level = *(volatile const int*)p.level;
    if (__syncthreads_or(MODE == I8_BOUND ? level == kI8Rejected : level != MODE)) return;
  }
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
  const int nseg = (p.nkb + P::SEG_KB - 1) / P::SEG_KB;
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
        for (int pl = 0; pl < P::PLANES && ok; ++pl) {
          const signed char* plane = isb ? p.B + pl * p.b_plane : p.A + pl * p.a_plane;
          const int k0 = seg * P::SEG_KB, k1 = min(p.nkb, k0 + P::SEG_KB);
          for (int pass = 0; pass < P::PASSES && ok; ++pass)
            for (int kb = k0; kb < k1; kb += P::blocks(pass), ++it) {
              const int s = it % I8_STAGES;
              if (it >= I8_STAGES && !mbar_wait(empty + 8 * s, (uint32_t)((it / I8_STAGES - 1) & 1), lim)) s_fail = 1;
              if (__any_sync(0xffffffffu, s_fail != 0)) {
                ok = false;
                break;
              }
              const int nd = P::digits(pass), blocks = min(P::blocks(pass), k1 - kb);
              const int kk = kb + sub / nd, dg = sub % nd;
              const long long block = MODE == I8_BOUND ? kk : (long long)kk * I8_S + dg;
              if (lane == 0) mbar_expect_tx(full + 8 * s, blocks * nd * S::SUB);
              __syncwarp();
              if (sub < blocks * nd)
                bulk_load(base + s * S::STAGE + dst, plane + ((block * 2 + kc) * rows + row0) * 16, bytes, full + 8 * s);
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
          for (int pl = 0; pl < P::PLANES && ok; ++pl) {
            const int k0 = seg * P::SEG_KB, k1 = min(p.nkb, k0 + P::SEG_KB);
            for (int pass = 0; pass < P::PASSES && ok; ++pass, ++u) {
              if (u > 0 && !mbar_wait(acc_empty, (uint32_t)((u - 1) & 1), lim)) ok = false;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              for (int kb = k0; ok && kb < k1; kb += P::blocks(pass), ++it) {
                const int s = it % I8_STAGES;
                if (s_fail || !mbar_wait(full + 8 * s, (uint32_t)((it / I8_STAGES) & 1), lim)) {
                  ok = false;
                  break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t stage = base + s * S::STAGE;
                if (pass == 0) i8_issue<BN, MODE, 0>(stage, tmem, kb == k0, k1 - kb);
                if constexpr (P::PASSES > 1)
                  if (pass == 1) i8_issue<BN, MODE, 1>(stage, tmem, kb == k0, k1 - kb);
                if constexpr (P::PASSES > 2)
                  if (pass == 2) i8_issue<BN, MODE, 2>(stage, tmem, kb == k0, k1 - kb);
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
      const int ea = MODE == I8_BOUND ? 0 : p.ea[r];
      Cx<double>* C = (f ? p.C[1] : p.C[0]) + (row_ok ? e : 0);
      for (int seg = 0; seg < nseg && ok; ++seg)
        for (int pl = 0; pl < P::PLANES && ok; ++pl)
          for (int pass = 0; pass < P::PASSES; ++pass, ++u) {
            const bool stop = __any_sync(0xffffffffu, s_fail != 0);
            if (!__all_sync(0xffffffffu, !stop && mbar_wait(acc_full, (uint32_t)(u & 1), lim))) {
              ok = false;
              s_fail = 1;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if constexpr (MODE == I8_BOUND) {
              int level = I8_PLAIN;
              const bool live = row_ok && p.amax[r] != 0;
#pragma unroll 1
              for (int c = 0; c < CH; c += 8) {
                int v[8];
                tmem_ld8(tmem + tlane + (uint32_t)(c0 + c), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 8; ++q)
                  if (v[q] < p.wide_line && live && n0 + c + q < p.N && p.bmax[n0 + c + q] != 0)
                    level = max(level, v[q] < p.reject_line ? kI8Rejected : (int)I8_WIDE);
              }
              if (level > *(volatile int*)p.level) atomicMax(p.level, level);
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              mbar_arrive(acc_empty);
              continue;
            }
            const bool first = seg == 0 && pl == 0 && pass == 0;
            // x = X 2^(e - 61); the last sum in units of 256^(14 - diagonal)
            const int unit = ea - 2 * I8_TOP + 8 * (15 - P::low(pass) - P::sums(pass));
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
                const long long x = P::sums(pass) == 1 ? (long long)v[0][q]
                                                       : ((((long long)v[0][q] << 8) + v[1][q]) * 65536) +
                                                             (((long long)v[2][q] << 8) + v[3][q]);
                const double y = scalbn((double)x, unit + p.eb[n0 + c + q]);
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
  if (threadIdx.x == 0 && s_fail) {
    record_status(p.status, QCL_TIMEOUT, (long long)blockIdx.x);
    if (MODE == I8_BOUND) atomicMax(p.level, kI8Rejected);
  }
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
__global__ void i8_row_max_kernel(I8Src a, unsigned long long* __restrict__ rowmax, int kper, const int* level) {
  if (*level == kI8Rejected) return;  // by an earlier panel (launch-uniform)
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

// Exponent of a row maximum (0 for a zero row), and the factors of
// x 2^(top - ex) in two exact steps (either alone stays in range).
__device__ __forceinline__ int i8_scale(double mx, int top, double& s1, double& s2) {
  int ex = 0;
  if (mx > 0.0 && !isinf(mx)) frexp(mx, &ex);
  const int sh = top - ex, sh1 = sh / 2;
  s1 = ldexp(1.0, sh1);
  s2 = ldexp(1.0, sh - sh1);
  return ex;
}

// Element k of a row, weighted.
__device__ __forceinline__ Cx<double> i8_element(const I8Src& a, const Cx<double>* X, int k) {
  const Cx<double> v = X[a.ld * k];
  const double w = a.w ? a.w[k % a.wmod] : 1.0;
  return cx<double>(v.x * w, v.y * w);
}

// The leading 7 bits of the larger part of every entry, relative to the power
// of two above the row maximum and rounded down; layout as the digits.  One
// thread per row and 16-wide K half.
__global__ void __launch_bounds__(256) i8_leading_kernel(I8Src a, const unsigned long long* __restrict__ rowmax,
                                                         signed char* __restrict__ out, int halves, int* level) {
  if (*(volatile const int*)level == kI8Rejected) return;
  const int r = blockIdx.x * 32 + (threadIdx.x & 31), f = r / a.rpad, e = r - f * a.rpad;
  const int half = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (half >= halves) return;
  const bool live = e < a.rows;
  const double mx = live ? __longlong_as_double((long long)rowmax[r]) : 0.0;
  double s1, s2;
  i8_scale(mx, 7, s1, s2);
  if (isinf(mx) && half == 0) atomicMax(level, kI8Rejected);
  const bool use = live && !isinf(mx);
  const Cx<double>* X = (f ? a.X[1] : a.X[0]) + e;
  unsigned q[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    q[g] = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = half * 16 + 4 * g + i;
      if (!use || k >= a.K) continue;
      const Cx<double> v = i8_element(a, X, k);
      q[g] |= (unsigned)__double2int_rz(fmax(fabs(v.x), fabs(v.y)) * s1 * s2) << (8 * i);
    }
  }
  *reinterpret_cast<uint4*>(out + ((long long)half * a.total + r) * 16) = make_uint4(q[0], q[1], q[2], q[3]);
}

// One thread per row and 16-wide K half: 16 values, their 3 x 16 integers, and
// 3 x 8 digit rows of 16 bytes.  A warp reads and writes 512 contiguous bytes.
__global__ void __launch_bounds__(256) i8_split_kernel(I8Src a, const unsigned long long* __restrict__ rowmax,
                                                       int* __restrict__ exps, signed char* __restrict__ out,
                                                       long long plane, int halves, const int* level) {
  if (*level == kI8Rejected) return;
  const int r = blockIdx.x * 32 + (threadIdx.x & 31), f = r / a.rpad, e = r - f * a.rpad;
  const int half = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (half >= halves) return;
  const bool live = e < a.rows;
  const double mx = live ? __longlong_as_double((long long)rowmax[r]) : 0.0;
  double s1, s2;
  const int ex = i8_scale(mx, I8_TOP, s1, s2);
  if (half == 0) exps[r] = ex;
  const Cx<double>* X = (f ? a.X[1] : a.X[0]) + e;
  long long xr[16], xi[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int k = half * 16 + i;
    Cx<double> v = cx<double>(0, 0);
    if (live && k < a.K) v = i8_element(a, X, k);
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

// Operand rows for m rows of a field of A and for n columns (whole tiles of every width).
static int i8_mpad(int m) { return ceil_div(m, I8_BM) * I8_BM; }
static int i8_bpad(int n) { return ceil_div(n, I8_MAXBN) * I8_MAXBN + I8_MAXBN; }

// The work area: the product's level, the row maxima of all rows, the exponents
// and the digits (or leading bits) of one panel of B and one of A.
struct I8Layout {
  int mpan, npan, mpans, npans;  // rows of a field and columns per panel, panels
  int rows, bpad;                // operand rows of a full panel of A (both fields) and of B
  int nkb;                       // K blocks (even)
  size_t level, amax, bmax, ea, eb, B, A, bytes;
};
static I8Layout i8_layout(int M, int fields, int N, int K, int mp, int np) {
  const auto panel = [](int n, int parts, int unit) { return std::min(n, ceil_div(ceil_div(n, parts), unit) * unit); };
  I8Layout l;
  l.mpan = panel(M, mp, I8_BM);
  l.npan = panel(N, np, I8_MAXBN);
  l.mpans = ceil_div(M, l.mpan);
  l.npans = ceil_div(N, l.npan);
  l.rows = fields * i8_mpad(l.mpan);
  l.bpad = i8_bpad(l.npan);
  l.nkb = ceil_div(K, 2 * I8_KB) * 2;
  size_t at = 0;
  const auto take = [&](size_t n) {
    const size_t r = at;
    at += (n + 255) / 256 * 256;
    return r;
  };
  const size_t row = 3 * (size_t)l.nkb * I8_KB * I8_S;  // digits; the leading bits take less
  l.level = take(sizeof(int));
  l.amax = take((size_t)l.mpans * l.rows * 8);
  l.bmax = take((size_t)l.npans * l.bpad * 8);
  l.ea = take((size_t)l.rows * 4);
  l.eb = take((size_t)l.bpad * 4);
  l.B = take(l.bpad * row);
  l.A = take(l.rows * row);
  l.bytes = at;
  return l;
}

size_t i8_work_bytes(int M, int fields, int N, int K, int panel_rows) {
  return i8_layout(M, fields, N, K, panel_rows > 0 ? ceil_div(M, panel_rows) : 1, 1).bytes;
}
size_t i8_least_bytes(int M, int fields, int N, int K) {
  return i8_layout(M, fields, N, K, ceil_div(M, I8_BM), ceil_div(N, I8_MAXBN)).bytes;
}

// Whether the product is large enough for the bound and the split to pay.  One
// iteration of a solve with one such map, FP64 tensor path / this one / this one
// rejecting the product (rows x K x columns):
//   1000 x 1152^2: 767 / 772 / 828 us, 384 x 2048^2: 820 / 782 / 860 us,
//   1024 x 2048^2: 1734 / 1149 / 1820 us, 2048 x 4096^2: 10.87 / 5.60 / 11.21 ms;
// beyond the lines 600 x 1152^2 (8e8): 578 us at best either way, 192 x 4096^2:
// 1299 / 1370 / 1486 us (few rows share the passes over B).
bool i8_worthwhile(int M, int fields, int N, int K) {
  return (double)M * fields * N * K >= 1e9 && (long long)M * fields >= 384 && N >= 64 && K >= 64;
}

template <int BN, int MODE> static int launch_i8_t(const I8Args& a, int sms, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(
        cudaFuncSetAttribute(i8_gemm_kernel<BN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, I8Shape<BN>::SMEM));
    configured = true;
  }
  const int tiles = a.mtiles * a.ntiles;
  i8_gemm_kernel<BN, MODE><<<std::min(tiles, sms), I8_THREADS, I8Shape<BN>::SMEM, st>>>(a);
  QCL_LAUNCH_CHECK("i8_gemm_kernel");
  return QCL_OK;
}

template <int BN> static int launch_i8_levels(const I8Args& a, int sms, cudaStream_t st) {
  const int s = launch_i8_t<BN, I8_PLAIN>(a, sms, st);
  return s ? s : launch_i8_t<BN, I8_WIDE>(a, sms, st);
}

static int i8_row_max(const I8Src& a, unsigned long long* rowmax, const int* level, cudaStream_t st) {
  QCL_CUDA_CHECK(cudaMemsetAsync(rowmax, 0, (size_t)a.total * sizeof(unsigned long long), st));
  const int rb = a.total / 32;
  const int ks = std::max(1, std::min(ceil_div(a.K, 64), 8 * 148 / rb));
  const int kper = ceil_div(a.K, ks);
  i8_row_max_kernel<<<dim3(rb, ceil_div(a.K, kper)), 256, 0, st>>>(a, rowmax, kper, level);
  QCL_LAUNCH_CHECK("i8_row_max_kernel");
  return QCL_OK;
}

// K blocks of leading bits.
static int i8_bound_blocks(int K) { return std::min(ceil_div(K, I8_KB), I8_BOUND_MAX_KB); }
static int i8_leading(const I8Src& a, const unsigned long long* rowmax, signed char* out, int* level, cudaStream_t st) {
  const int halves = 2 * i8_bound_blocks(a.K);
  i8_leading_kernel<<<dim3(a.total / 32, ceil_div(halves, 8)), 256, 0, st>>>(a, rowmax, out, halves, level);
  QCL_LAUNCH_CHECK("i8_leading_kernel");
  return QCL_OK;
}

static int i8_split(const I8Src& a, const unsigned long long* rowmax, int* exps, signed char* out, int nkb,
                    const int* level, cudaStream_t st) {
  const long long plane = (long long)nkb * I8_S * 2 * a.total * 16;
  i8_split_kernel<<<dim3(a.total / 32, ceil_div(2 * nkb, 8)), 256, 0, st>>>(a, rowmax, exps, out, plane, 2 * nkb,
                                                                            level);
  QCL_LAUNCH_CHECK("i8_split_kernel");
  return QCL_OK;
}

// The product, unless *(int*)work is kI8Rejected afterwards: then C is as it
// was, and the caller's launch on the FP64 tensor path takes over
// (GemmArgs::i8_level).
int launch_i8_gemm(int M, int fields, int N, int K, const void* const* A, long long lda, const double* w, int wmod,
                   const void* B, long long ldb, void* const* C, long long ldc, double alpha, double beta, void* work,
                   size_t work_bytes, int* status, cudaStream_t st) {
  const int sms = sm_count();
  // panels: rows of A (one field) and columns of B that the work area holds
  int mp = 1, np = 1;
  I8Layout l = i8_layout(M, fields, N, K, mp, np);
  while (l.bytes > work_bytes) {
    if (l.rows >= l.bpad && l.mpan > I8_BM) ++mp;
    else if (l.npan > I8_MAXBN) ++np;
    else if (l.mpan > I8_BM) ++mp;
    else {
      set_last_error("i8 product: work area of %zu bytes is too small", work_bytes);
      return QCL_UNSUPPORTED;
    }
    l = i8_layout(M, fields, N, K, mp, np);
  }
  char* const base = (char*)work;
  int* const level = (int*)(base + l.level);
  int *const ea = (int*)(base + l.ea), *const eb = (int*)(base + l.eb);
  signed char *const Bd = (signed char*)(base + l.B), *const Ad = (signed char*)(base + l.A);
  QCL_CUDA_CHECK(cudaMemsetAsync(level, 0, sizeof(int), st));
  int s;
  for (int bound = 1; bound >= 0; --bound)  // the bound of every panel before the first digit of C
    for (int j = 0; j < l.npans; ++j) {
      const int n0 = j * l.npan, n = std::min(l.npan, N - n0), bpad = i8_bpad(n);
      unsigned long long* const bmax = (unsigned long long*)(base + l.bmax) + (size_t)j * l.bpad;
      const I8Src bs{{(const Cx<double>*)B + n0, nullptr}, ldb, nullptr, 1, n, bpad, bpad, K};
      if (bound && (s = i8_row_max(bs, bmax, level, st))) return s;
      if ((s = bound ? i8_leading(bs, bmax, Bd, level, st) : i8_split(bs, bmax, eb, Bd, l.nkb, level, st))) return s;
      for (int i = 0; i < l.mpans; ++i) {
        const int m0 = i * l.mpan, m = std::min(l.mpan, M - m0), mpad = i8_mpad(m), rows = fields * mpad;
        unsigned long long* const amax = (unsigned long long*)(base + l.amax) + (size_t)i * l.rows;
        const I8Src as{{(const Cx<double>*)A[0] + m0, fields > 1 ? (const Cx<double>*)A[1] + m0 : nullptr}, lda, w, wmod,
                       m, mpad, rows, K};
        if (bound && j == 0 && (s = i8_row_max(as, amax, level, st))) return s;
        if (j == 0 || l.mpans > 1)
          if ((s = bound ? i8_leading(as, amax, Ad, level, st) : i8_split(as, amax, ea, Ad, l.nkb, level, st)))
            return s;
        I8Args g{};
        g.A = Ad;
        g.B = Bd;
        g.a_plane = (long long)l.nkb * I8_S * 2 * rows * 16;
        g.b_plane = (long long)l.nkb * I8_S * 2 * bpad * 16;
        g.a_rows = rows;
        g.b_rows = bpad;
        g.nkb = bound ? i8_bound_blocks(K) : l.nkb;
        g.mtiles = rows / I8_BM;
        g.M = m;
        g.mpad = mpad;
        g.N = n;
        g.ea = ea;
        g.eb = eb;
        g.amax = amax;
        g.bmax = bmax;
        g.level = level;
        g.wide_line = (int)ceil(16384 * sqrt((double)K) / 100);
        g.reject_line = (int)ceil(16384 * sqrt((double)K) / 1500);
        for (int f = 0; f < fields; ++f) g.C[f] = (Cx<double>*)C[f] + m0 + ldc * n0;
        g.ldc = ldc;
        g.alpha = alpha;
        g.beta = beta;
        g.status = status;
        const int bn = bound ? 128 : i8_pick_bn(g.mtiles, n, sms);
        g.ntiles = ceil_div(n, bn);
        if (bound) s = launch_i8_t<128, I8_BOUND>(g, sms, st);
        else if (bn == 128) s = launch_i8_levels<128>(g, sms, st);
        else if (bn == 112) s = launch_i8_levels<112>(g, sms, st);
        else if (bn == 96) s = launch_i8_levels<96>(g, sms, st);
        else s = launch_i8_levels<64>(g, sms, st);
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
