// Energy shifts and the static self-energy contractions.
//
// Shift: apply_energy_shift! (numerics/optimized/production_cache.jl:300-325)
//   Y[e] = valid[e] ? ((l == r || th == 0) ? X[l] : (1-th) X[l] + th X[r]) : 0
// Contractions (production_static_contraction, production_operators.jl:
// 402-658), S = beta S + alpha q K[wk G]:
//   momentum independent: X[e,(c,d)] = sum_m' wk G[e,m',c,d]; Y = B X;
//                         S[e,m,(a,b)] broadcast over m;
//   dense:                S[e,(m,a,b)] = sum_(m',c,d) M wk[m'] G[e,(m',c,d)];
//   separable IFR:        S = left * (radial * (wk .* (right * G)));
//   low rank:             S = left * (right_adjoint * (wk .* G));
//   separable sum:        S[e,m,(a,b)] = sum_i sum_(c,d) block_i[(a,b),(c,d)]
//                                        sum_m' radial_i[m,m'] wk[m'] G[e,m',c,d].
// Every stage is one call of a tiled complex GEMM whose operand and output
// index maps are strided views of the E-fastest fields: the energy axis is the
// GEMM's M dimension, so all A loads and C stores are coalesced along E.
#include "kernels.cuh"

namespace qcl {

// ---------------------------------------------------------------------------
template <typename R>
__global__ void shift_kernel(int NE, long long ncols, const int* __restrict__ left, const int* __restrict__ right,
                             const double* __restrict__ theta, const unsigned char* __restrict__ valid,
                             const Cx<R>* __restrict__ X, Cx<R>* __restrict__ Y) {
  const long long n = (long long)NE * ncols;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(i % NE);
    const long long base = i - e;
    Cx<R> v = cx<R>(0, 0);
    if (valid[e]) {
      const int l = left[e], r = right[e];
      const double th = theta[e];
      if (l == r || th == 0.0) {
        v = X[base + l];
      } else {
        const Cx<R> a = X[base + l], b = X[base + r];
        v = cx<R>((R)((1 - th) * a.x + th * b.x), (R)((1 - th) * a.y + th * b.y));
      }
    }
    Y[i] = v;
  }
}

static unsigned grid_cap(long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  const long long cap = 148 * 16;
  return (unsigned)(g < cap ? (g > 0 ? g : 1) : cap);
}

int launch_shift(int precision, int NE, long long ncols, const ShiftPlanDev& plan, const void* X, void* Y,
                 cudaStream_t st) {
  const long long n = (long long)NE * ncols;
  if (precision == QCL_C128)
    shift_kernel<double><<<grid_cap(n, 256), 256, 0, st>>>(NE, ncols, plan.left, plan.right, plan.theta, plan.valid,
                                                          (const Cx<double>*)X, (Cx<double>*)Y);
  else
    shift_kernel<float><<<grid_cap(n, 256), 256, 0, st>>>(NE, ncols, plan.left, plan.right, plan.theta, plan.valid,
                                                         (const Cx<float>*)X, (Cx<float>*)Y);
  QCL_LAUNCH_CHECK("shift_kernel");
  return QCL_OK;
}

// Y = a X(eps + d1) + b X(eps + d2): two shifts of the same field combined in
// one pass (the linear combination the thermal-LO self-energy contracts,
// production_operators.jl:1107-1163, formed before the contraction).
template <typename R>
__global__ void shift_pair_kernel(int NE, long long ncols, ShiftPlanDev p1, ShiftPlanDev p2, double a, double b,
                                  const Cx<R>* __restrict__ X, Cx<R>* __restrict__ Y) {
  const long long n = (long long)NE * ncols;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(i % NE);
    const long long base = i - e;
    double vx = 0, vy = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const ShiftPlanDev& pl = s == 0 ? p1 : p2;
      const double c = s == 0 ? a : b;
      if (!pl.valid[e]) continue;
      const int l = pl.left[e], r = pl.right[e];
      const double th = pl.theta[e];
      double ux, uy;
      if (l == r || th == 0.0) {
        const Cx<R> q = X[base + l];
        ux = q.x;
        uy = q.y;
      } else {
        const Cx<R> ql = X[base + l], qr = X[base + r];
        ux = (1 - th) * ql.x + th * qr.x;
        uy = (1 - th) * ql.y + th * qr.y;
      }
      vx += c * ux;
      vy += c * uy;
    }
    Y[i] = cx<R>((R)vx, (R)vy);
  }
}

int launch_shift_pair(int precision, int NE, long long ncols, const ShiftPlanDev& p1, const ShiftPlanDev& p2, double a,
                      double b, const void* X, void* Y, cudaStream_t st) {
  const long long n = (long long)NE * ncols;
  if (precision == QCL_C128)
    shift_pair_kernel<double><<<grid_cap(n, 256), 256, 0, st>>>(NE, ncols, p1, p2, a, b, (const Cx<double>*)X,
                                                               (Cx<double>*)Y);
  else
    shift_pair_kernel<float><<<grid_cap(n, 256), 256, 0, st>>>(NE, ncols, p1, p2, a, b, (const Cx<float>*)X,
                                                              (Cx<float>*)Y);
  QCL_LAUNCH_CHECK("shift_pair_kernel");
  return QCL_OK;
}

// build_shift_plan (production_cache.jl:258-290), 0-based, on the host.
int build_shift_plan_host(int NE, const double* eps, double delta, int* left, int* right, double* theta,
                          unsigned char* valid) {
  if (NE < 2 || !isfinite(delta)) {
    set_last_error("shift plan: at least two nodes and a finite displacement are required");
    return QCL_ARG;
  }
  for (int e = 1; e < NE; ++e)
    if (!(eps[e] > eps[e - 1]) || !isfinite(eps[e])) {
      set_last_error("energy nodes must be finite and strictly increasing");
      return QCL_ARG;
    }
  int j = 0;
  for (int e = 0; e < NE; ++e) {
    const double target = eps[e] + delta;
    left[e] = right[e] = 0;
    theta[e] = 0.0;
    valid[e] = 0;
    if (target < eps[0] || target > eps[NE - 1]) continue;
    if (target == eps[NE - 1]) {
      left[e] = right[e] = NE - 1;
      valid[e] = 1;
      continue;
    }
    while (j < NE - 2 && eps[j + 1] <= target) ++j;
    left[e] = j;
    right[e] = j + 1;
    theta[e] = (target - eps[j]) / (eps[j + 1] - eps[j]);
    valid[e] = 1;
  }
  return QCL_OK;
}

// ---------------------------------------------------------------------------
// Momentum reduction: X[e + NE q] = sum_m' wk[m'] G[e + NE (m' + Nk q)]
// ---------------------------------------------------------------------------
template <typename R>
__global__ void momentum_sum_kernel(int NE, int Nk, int NQ, const double* __restrict__ wk, const Cx<R>* G0,
                                    const Cx<R>* G1, Cx<R>* X0, Cx<R>* X1) {
  const Cx<R>* __restrict__ G = blockIdx.y ? G1 : G0;
  Cx<R>* __restrict__ X = blockIdx.y ? X1 : X0;
  const long long n = (long long)NE * NQ;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(i % NE);
    const long long q = i / NE;
    double sx = 0, sy = 0;
#pragma unroll 8
    for (int mp = 0; mp < Nk; ++mp) {
      const Cx<R> g = G[(size_t)e + (size_t)NE * ((size_t)mp + (size_t)Nk * q)];
      sx += wk[mp] * (double)g.x;
      sy += wk[mp] * (double)g.y;
    }
    X[i] = cx<R>((R)sx, (R)sy);
  }
}

// ---------------------------------------------------------------------------
// Complex GEMM over strided views, of one or two fields:
//   C[e, j] (bcast copies) = alpha * sum_k A[e,k] w(k,b) B[j,k] + beta * C
//   A[e,k] = A[f][e + lda k + a_b b],  B[j,k] = B[j + ldb k + b_b b],
//   C[e,j] = C[f][e + ldc j + c_b b + bcast_stride r], r < bcast,
// b < batch, f < fields.
// ---------------------------------------------------------------------------
template <typename R> struct GemmArgs {
  int M, Nout, K, batch;
  int fields = 1;
  const Cx<R>* A[2];
  long long lda, a_b;
  const double* wk;  // optional weight wk[k % wk_mod]
  int wk_mod;
  const double* wb;  // optional weight wb[b]
  const Cx<R>* B;
  long long ldb, b_b;
  Cx<R>* C[2];
  long long ldc, c_b;
  int bcast;
  long long bcast_stride;
  double alpha, beta;
  // tile order: 0 = row tiles fastest (the CTAs in flight share B tiles),
  // 1 = column tiles fastest (they share A tiles: an A larger than L2 is
  // read once); set by launch_gemm for complex128
  int cols_fastest;
  // complex128: run only if the integer path rejected the product (NULL: always)
  const int* i8_level;
};

template <typename R> __device__ __forceinline__ void gemm_store(const GemmArgs<R>& p, Cx<R>* C, int e, int j, Cx<R> acc) {
  const double vx = p.alpha * (double)acc.x, vy = p.alpha * (double)acc.y;
  for (int r = 0; r < p.bcast; ++r) {
    const size_t idx = (size_t)e + (size_t)p.ldc * j + (size_t)p.bcast_stride * r;
    if (p.beta == 0.0) {
      C[idx] = cx<R>((R)vx, (R)vy);
    } else {
      const Cx<R> o = C[idx];
      C[idx] = cx<R>((R)(p.beta * o.x + vx), (R)(p.beta * o.y + vy));
    }
  }
}

// complex64: CUDA cores.  Output tile GE x GJ per CTA of GT threads: a 16 x
// (GT / 16) thread grid, each thread GE/16 x GJ/(GT/16) outputs.  The next K
// block is fetched into registers while the current one is multiplied, all
// its loads in flight at once (loop by loop they were a chain of load
// latencies: 383 x 256 x 256 took 54 us for 0.2 GFLOP).
constexpr int GK = 16;
template <int GE, int GJ, int GT> __global__ void __launch_bounds__(GT) gemm_kernel(const __grid_constant__ GemmArgs<float> p) {
  using R = float;
  constexpr int TJ = GT / 16, NI = GE / 16, NU = GJ / TJ;
  constexpr int NA = GE * GK / GT, NB = GJ * GK / GT;
  static_assert(GE % 16 == 0 && GJ % TJ == 0 && NA * GT == GE * GK && NB * GT == GJ * GK, "tile shape");
  __shared__ Cx<R> As[2][GK][GE];
  __shared__ Cx<R> Bs[2][GK][GJ];
  const int f = blockIdx.z / p.batch, b = blockIdx.z - f * p.batch;
  const int e0 = blockIdx.x * GE, j0 = blockIdx.y * GJ;
  const int te = threadIdx.x % 16, tj = threadIdx.x / 16;
  const double wbb = p.wb ? p.wb[b] : 1.0;
  const Cx<R>* A = (f ? p.A[1] : p.A[0]) + (size_t)p.a_b * b;
  const Cx<R>* B = p.B + (size_t)p.b_b * b;
  Cx<R>* C = (f ? p.C[1] : p.C[0]) + (size_t)p.c_b * b;
  Cx<R> acc[NI][NU], ra[NA], rb[NB];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int u = 0; u < NU; ++u) acc[i][u] = cx<R>(0, 0);
  double rw[NA];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int idx = threadIdx.x + q * GT, e = e0 + idx % GE, k = k0 + idx / GE;
      const bool ok = e < p.M && k < p.K;
      ra[q] = ok ? A[(size_t)e + (size_t)p.lda * k] : cx<R>(0, 0);
      rw[q] = p.wk && ok ? wbb * p.wk[k % p.wk_mod] : wbb;
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int idx = threadIdx.x + q * GT, j = j0 + idx % GJ, k = k0 + idx / GJ;
      rb[q] = j < p.Nout && k < p.K ? B[(size_t)j + (size_t)p.ldb * k] : cx<R>(0, 0);
    }
  };
  fetch(0);
  for (int k0 = 0, s = 0; k0 < p.K; k0 += GK, s ^= 1) {
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int idx = threadIdx.x + q * GT;
      As[s][idx / GE][idx % GE] = rw[q] == 1.0 ? ra[q] : cx<R>((R)(rw[q] * ra[q].x), (R)(rw[q] * ra[q].y));
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int idx = threadIdx.x + q * GT;
      Bs[s][idx / GJ][idx % GJ] = rb[q];
    }
    __syncthreads();  // stage s is complete; its other half was read before the last barrier
    if (k0 + GK < p.K) fetch(k0 + GK);
#pragma unroll
    for (int kl = 0; kl < GK; ++kl) {
      Cx<R> a[NI], bb[NU];
#pragma unroll
      for (int i = 0; i < NI; ++i) a[i] = As[s][kl][te + 16 * i];
#pragma unroll
      for (int u = 0; u < NU; ++u) bb[u] = Bs[s][kl][tj + TJ * u];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int u = 0; u < NU; ++u) cfma(acc[i][u], a[i], bb[u]);
    }
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int e = e0 + te + 16 * i;
    if (e >= p.M) continue;
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      const int j = j0 + tj + TJ * u;
      if (j < p.Nout) gemm_store<R>(p, C, e, j, acc[i][u]);
    }
  }
}

// Wider tiles while they leave two CTAs per SM; narrower ones, down to 32 x 16,
// fill the GPU at the sizes where a launch would otherwise be a few CTAs.
static int launch_gemm(const GemmArgs<float>& a, cudaStream_t st) {
  if (a.M <= 0 || a.Nout <= 0 || a.batch <= 0) return QCL_OK;
  const int z = a.batch * a.fields;
  auto ctas = [&](int ge, int gj) { return (long long)((a.M + ge - 1) / ge) * ((a.Nout + gj - 1) / gj) * z; };
  if (a.Nout > 32 && ctas(64, 64) >= 2 * 148) {
    gemm_kernel<64, 64, 256><<<dim3((a.M + 63) / 64, (a.Nout + 63) / 64, z), 256, 0, st>>>(a);
  } else if (a.Nout > 16 && ctas(64, 32) >= 2 * 148) {
    gemm_kernel<64, 32, 256><<<dim3((a.M + 63) / 64, (a.Nout + 31) / 32, z), 256, 0, st>>>(a);
  } else {
    gemm_kernel<32, 16, 128><<<dim3((a.M + 31) / 32, (a.Nout + 15) / 16, z), 128, 0, st>>>(a);
  }
  QCL_LAUNCH_CHECK("gemm_kernel");
  return QCL_OK;
}

// ---------------------------------------------------------------------------
// complex128: the FP64 tensor path (mma.sync m8n8k4 f64).  CTA: BM (e) x 32 (j)
// outputs on BM / (8 TR) x 2 warps; warp (wm, wn) owns 8 TR rows and 16 columns
// as TR x 2 tiles of 8 x 8, each accumulated as four real
// products (Re C += Ar Br - Ai Bi, Im C += Ar Bi + Ai Br); tiles past the last
// column are skipped.  K advances by 16 through 2 or 3 cp.async stages; shared
// rows are padded to a stride of 2 (mod 8) 16-byte units so the fragment
// loads of a quarter warp hit 8 distinct bank groups.  Fragment layouts
// (m8n8k4, f64): A lane l holds (l / 4, l % 4), B holds (l % 4, l / 4), C holds
// (l / 4, 2 (l % 4) + i).
// ---------------------------------------------------------------------------
constexpr int DM_BN = 32, DM_BK = 16;
constexpr int DM_BPAD = DM_BN + 2;
// at least four warps, one per scheduler: each has a quarter of the FP64 rate
template <int BM_> struct DmShape {
  static constexpr int BM = BM_, TR = BM == 32 ? 2 : 4, WM = BM / (8 * TR), THREADS = 64 * WM, APAD = BM + 2;
  static constexpr int STAGES = BM == 32 ? 3 : 2;  // CTAs per SM: 2, 4, 4
  static constexpr size_t SMEM =
      STAGES * (DM_BK * (APAD + DM_BPAD) * sizeof(Cx<double>) + DM_BK * sizeof(double));
};

__device__ __forceinline__ void dm_cp16(Cx<double>* dst, const Cx<double>* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int BM>
__global__ void __launch_bounds__(DmShape<BM>::THREADS, BM == 128 ? 2 : 4) dmma_gemm_kernel(const __grid_constant__ GemmArgs<double> p) {
  using S = DmShape<BM>;
  constexpr int TR = S::TR, WM = S::WM, ST = S::STAGES;
  if (p.i8_level && *p.i8_level != kI8Rejected) return;  // launch-uniform
  extern __shared__ __align__(16) unsigned char dm_raw[];
  Cx<double>* As = reinterpret_cast<Cx<double>*>(dm_raw);            // [ST][DM_BK][APAD]
  Cx<double>* Bs = As + ST * DM_BK * S::APAD;                         // [ST][DM_BK][DM_BPAD]
  double* ws = reinterpret_cast<double*>(Bs + ST * DM_BK * DM_BPAD);  // [ST][DM_BK]
  const int m0 = (p.cols_fastest ? blockIdx.y : blockIdx.x) * S::BM;
  const int n0 = (p.cols_fastest ? blockIdx.x : blockIdx.y) * DM_BN;
  const int f = blockIdx.z / p.batch, b = blockIdx.z - f * p.batch;
  const double wbb = p.wb ? p.wb[b] : 1.0;
  const Cx<double>* A = (f ? p.A[1] : p.A[0]) + (size_t)p.a_b * b;
  const Cx<double>* B = p.B + (size_t)p.b_b * b;
  Cx<double>* C = (f ? p.C[1] : p.C[0]) + (size_t)p.c_b * b;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp % WM, wn = warp / WM;
  const int lr = lane >> 2, lc = lane & 3;
  const bool col_in[2] = {n0 + wn * 16 < p.Nout, n0 + wn * 16 + 8 < p.Nout};  // warp-uniform
  double cr[TR][2][2], ci[TR][2][2];
#pragma unroll
  for (int t = 0; t < TR; ++t)
#pragma unroll
    for (int u = 0; u < 2; ++u) cr[t][u][0] = cr[t][u][1] = ci[t][u][0] = ci[t][u][1] = 0.0;

  const int nkb = (p.K + DM_BK - 1) / DM_BK;
  auto load = [&](int kb, int s) {
    const int k0 = kb * DM_BK;
    Cx<double>* as = As + s * DM_BK * S::APAD;
    Cx<double>* bs = Bs + s * DM_BK * DM_BPAD;
#pragma unroll
    for (int i = threadIdx.x; i < DM_BK * S::BM; i += S::THREADS) {
      const int kk = i / S::BM, el = i % S::BM;
      const int k = k0 + kk, e = m0 + el;
      const bool ok = k < p.K && e < p.M;
      dm_cp16(as + kk * S::APAD + el, ok ? A + (size_t)e + (size_t)p.lda * k : A, ok);
    }
#pragma unroll
    for (int i = threadIdx.x; i < DM_BK * DM_BN; i += S::THREADS) {
      const int kk = i / DM_BN, jl = i % DM_BN;
      const int k = k0 + kk, j = n0 + jl;
      const bool ok = k < p.K && j < p.Nout;
      dm_cp16(bs + kk * DM_BPAD + jl, ok ? B + (size_t)j + (size_t)p.ldb * k : B, ok);
    }
    if (threadIdx.x < DM_BK) {
      const int k = k0 + threadIdx.x;
      ws[s * DM_BK + threadIdx.x] = (k < p.K && p.wk) ? wbb * p.wk[k % p.wk_mod] : wbb;
    }
  };

  // one commit group per stage, empty past the last block, so that the wait
  // counts stages
#pragma unroll
  for (int q = 0; q < ST - 1; ++q) {
    if (q < nkb) load(q, q);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kb = 0; kb < nkb; ++kb) {
    const int s = kb % ST;
    // the stage being refilled was released by the barrier at the end of iteration kb - 1
    if (kb + ST - 1 < nkb) load(kb + ST - 1, (kb + ST - 1) % ST);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 1) : "memory");
    __syncthreads();
    const Cx<double>* as = As + s * DM_BK * S::APAD;
    const Cx<double>* bs = Bs + s * DM_BK * DM_BPAD;
    if (col_in[0]) {
#pragma unroll
      for (int c = 0; c < DM_BK / 4; ++c) {
        const int kk = 4 * c + lc;
        const double w = ws[s * DM_BK + kk];
        double ar[TR], ai[TR], nai[TR], br[2], bi[2];
#pragma unroll
        for (int t = 0; t < TR; ++t) {
          const Cx<double> a = as[kk * S::APAD + wm * 8 * TR + t * 8 + lr];
          ar[t] = a.x * w;
          ai[t] = a.y * w;
          nai[t] = -ai[t];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const Cx<double> bv = bs[kk * DM_BPAD + wn * 16 + u * 8 + lr];
          br[u] = bv.x;
          bi[u] = bv.y;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (!col_in[u]) continue;
#pragma unroll
          for (int t = 0; t < TR; ++t) {
            dmma(cr[t][u], ar[t], br[u]);
            dmma(cr[t][u], nai[t], bi[u]);
            dmma(ci[t][u], ar[t], bi[u]);
            dmma(ci[t][u], ai[t], br[u]);
          }
        }
      }
    }
    __syncthreads();  // every warp is done with stage s before it is refilled
  }
#pragma unroll
  for (int t = 0; t < TR; ++t) {
    const int e = m0 + wm * 8 * TR + t * 8 + lr;
    if (e >= p.M) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = n0 + wn * 16 + u * 8 + 2 * lc + i;
        if (j < p.Nout) gemm_store<double>(p, C, e, j, cx<double>(cr[t][u][i], ci[t][u][i]));
      }
  }
}

template <int BM> static int launch_dmma_t(const GemmArgs<double>& a, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(dmma_gemm_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)DmShape<BM>::SMEM));
    configured = true;
  }
  const int mt = (a.M + BM - 1) / BM, nt = (a.Nout + DM_BN - 1) / DM_BN, z = a.batch * a.fields;
  const dim3 grid = a.cols_fastest ? dim3(nt, mt, z) : dim3(mt, nt, z);
  dmma_gemm_kernel<BM><<<grid, DmShape<BM>::THREADS, DmShape<BM>::SMEM, st>>>(a);
  QCL_LAUNCH_CHECK("dmma_gemm_kernel");
  return QCL_OK;
}

// Tile height by the rows the busiest SM works through (the FP64 rate is the
// bound): 64 x 48^2 x 48^2 436 -> 183 us with 32 rows, 383 x 2048^2 670 -> 515 us
// with 64, where 128 rows leave SMs without a tile.  Shorter tiles load more
// per product, hence their handicap.
static int launch_gemm(const GemmArgs<double>& args, cudaStream_t st) {
  GemmArgs<double> a = args;
  if (a.M <= 0 || a.Nout <= 0 || a.batch <= 0) return QCL_OK;
  const int nt = (a.Nout + DM_BN - 1) / DM_BN, z = a.batch * a.fields;
  auto ctas = [&](int bm) { return (long long)((a.M + bm - 1) / bm) * nt * z; };
  // the larger operand is read once: an A larger than B and than L2 streams
  // with the column tiles fastest
  const int mt = (a.M + 127) / 128;
  a.cols_fastest = a.M > a.Nout && (size_t)a.M * a.K * sizeof(Cx<double>) > ((size_t)96 << 20) && mt <= 65535;
  auto rows = [&](int bm) { return (double)((ctas(bm) + 147) / 148 * bm); };
  const double r128 = rows(128), r64 = 1.07 * rows(64), r32 = 1.2 * rows(32);
  if (r128 <= r64 && r128 <= r32) return launch_dmma_t<128>(a, st);
  if (r64 <= r32) return launch_dmma_t<64>(a, st);
  return launch_dmma_t<32>(a, st);
}

// ---------------------------------------------------------------------------
// Contraction dispatch
// ---------------------------------------------------------------------------
constexpr size_t kOperandAlign = 256;  // of tensor-core operands behind the intermediate (a tensor map needs 16)

// Whether a complex128 product goes to the integer path: large enough, and
// the operator's work area holds its smallest panels.
static bool takes_i8(const KernelOpDev& op, int M, int fields, int N, int K) {
  return op.i8_work && i8_worthwhile(M, fields, N, K) && op.i8_bytes >= i8_least_bytes(M, fields, N, K);
}

// One or two fields G[f] -> S[f].  work holds contraction_work_elems elements;
// with two fields, work2 as many again.
template <typename R>
static int contraction_t(const KernelOpDev& op, int NE, int Nk, int N, const double* wk, int fields,
                         const void* const* Gv, void* const* Sv, double alpha_q, double beta, void* work, void* work2,
                         cudaStream_t st) {
  const int N2 = N * N;
  const long long NEl = NE;
  const Cx<R>* const G[2] = {(const Cx<R>*)Gv[0], fields > 1 ? (const Cx<R>*)Gv[1] : nullptr};
  Cx<R>* const S[2] = {(Cx<R>*)Sv[0], fields > 1 ? (Cx<R>*)Sv[1] : nullptr};
  Cx<R>* const T[2] = {(Cx<R>*)work, (Cx<R>*)work2};
  if (op.kind == QCL_KERNEL_MOMENTUM_INDEPENDENT) {
    const long long n = NEl * N2;  // T[f]: NE * N2
    momentum_sum_kernel<R><<<dim3(grid_cap(n, 256), fields), 256, 0, st>>>(NE, Nk, N2, wk, G[0], G[1], T[0], T[1]);
    QCL_LAUNCH_CHECK("momentum_sum_kernel");
    GemmArgs<R> g{};
    g.M = NE; g.Nout = N2; g.K = N2; g.batch = 1; g.fields = fields;
    g.B = (const Cx<R>*)op.block; g.ldb = N2;
    g.ldc = NEl * Nk; g.bcast = Nk; g.bcast_stride = NEl;
    g.lda = NEl;
    g.alpha = alpha_q; g.beta = beta;
    for (int f = 0; f < 2; ++f) {
      g.A[f] = T[f];
      g.C[f] = S[f];
    }
    return launch_gemm(g, st);
  }
  if (op.kind == QCL_KERNEL_DENSE) {
    const int Nc = Nk * N2;
    if (sizeof(R) == 4 && op.tc_bop) {  // complex64 fields: tensor cores (scaled FP16 hi/lo)
      for (int f = 0; f < fields; ++f)
        if (int s = launch_tc_dense_contraction(NE, Nc, op.tc_bop, Gv[f], Sv[f], alpha_q, beta, (float*)work, op.status, st))
          return s;
      return QCL_OK;
    }
    GemmArgs<R> g{};
    if (sizeof(R) == 8 && takes_i8(op, NE, fields, Nc, Nc)) {
      if (int s = launch_i8_gemm(NE, fields, Nc, Nc, Gv, NEl, wk, Nk, op.matrix, Nc, Sv, NEl, alpha_q, beta, op.i8_work,
                                 op.i8_bytes, op.status, st))
        return s;
      g.i8_level = (const int*)op.i8_work;
    }
    g.M = NE; g.Nout = Nc; g.K = Nc; g.batch = 1; g.fields = fields;
    g.lda = NEl; g.wk = wk; g.wk_mod = Nk;
    g.B = (const Cx<R>*)op.matrix; g.ldb = Nc;
    g.ldc = NEl; g.bcast = 1;
    g.alpha = alpha_q; g.beta = beta;
    for (int f = 0; f < 2; ++f) {
      g.A[f] = G[f];
      g.C[f] = S[f];
    }
    return launch_gemm(g, st);
  }
  if (op.kind == QCL_KERNEL_IFR) {
    const int J = op.J;  // T[e + NE (j + J m')], then F[e + NE (j + J m)] behind it
    const size_t half = (size_t)NE * J * Nk;
    int s;
    GemmArgs<R> g{}, h{}, f{};
    // stage 1, batch m': T = wk[m'] right * G_m'
    g.M = NE; g.Nout = J; g.K = N2; g.batch = Nk; g.fields = fields;
    g.lda = NEl * Nk; g.a_b = NEl; g.wb = wk;
    g.B = (const Cx<R>*)op.right; g.ldb = J;
    g.ldc = NEl; g.c_b = NEl * J; g.bcast = 1;
    g.alpha = 1.0; g.beta = 0.0;
    // stage 2, batch j: F[., j, m] = sum_m' radial[m, m'] T[., j, m']
    h.M = NE; h.Nout = Nk; h.K = Nk; h.batch = J; h.fields = fields;
    h.lda = NEl * J; h.a_b = NEl;
    h.B = (const Cx<R>*)op.radial; h.ldb = Nk;
    h.ldc = NEl * J; h.c_b = NEl; h.bcast = 1;
    h.alpha = 1.0; h.beta = 0.0;
    // stage 3, batch m: S[., m, p] = alpha q sum_j left[p, j] F[., j, m] + beta S
    f.M = NE; f.Nout = N2; f.K = J; f.batch = Nk; f.fields = fields;
    f.lda = NEl; f.a_b = NEl * J;
    f.B = (const Cx<R>*)op.left; f.ldb = N2;
    f.ldc = NEl * Nk; f.c_b = NEl; f.bcast = 1;
    f.alpha = alpha_q; f.beta = beta;
    for (int q = 0; q < 2; ++q) {
      Cx<R>* F = T[q] ? T[q] + half : nullptr;
      g.A[q] = G[q];
      g.C[q] = T[q];
      h.A[q] = T[q];
      h.C[q] = F;
      f.A[q] = F;
      f.C[q] = S[q];
    }
    if ((s = launch_gemm(g, st))) return s;
    if ((s = launch_gemm(h, st))) return s;
    return launch_gemm(f, st);
  }
  if (op.kind == QCL_KERNEL_LOW_RANK) {
    // LowRankProductionKernel (production_operators.jl:597-658):
    //   T[e, r] = sum_q right_adjoint[r, q] wk[q % Nk] G[e, q]      (NE x rank)
    //   S[e, q] = alpha q^K sum_r left[q, r] T[e, r] + beta S[e, q]
    const int Nc = Nk * N2, r = op.J;
    GemmArgs<R> g{}, f{};
    g.M = NE; g.Nout = r; g.K = Nc; g.batch = 1; g.fields = fields;
    g.lda = NEl; g.wk = wk; g.wk_mod = Nk;
    g.B = (const Cx<R>*)op.right; g.ldb = r;
    g.ldc = NEl; g.bcast = 1;
    g.alpha = 1.0; g.beta = 0.0;
    f.M = NE; f.Nout = Nc; f.K = r; f.batch = 1; f.fields = fields;
    f.lda = NEl;
    f.B = (const Cx<R>*)op.left; f.ldb = Nc;
    f.ldc = NEl; f.bcast = 1;
    f.alpha = alpha_q; f.beta = beta;
    for (int q = 0; q < 2; ++q) {
      g.A[q] = G[q];
      g.C[q] = T[q];
      f.A[q] = T[q];
      f.C[q] = S[q];
    }
    if (int s = launch_gemm(g, st)) return s;
    return launch_gemm(f, st);
  }
  if (op.kind == QCL_KERNEL_SEPARABLE_SUM) {
    // K(m,m') = sum_i radial_i(m,m') block_i: a Kronecker sum of J terms (the
    // exact LO form sum_h R_h(m,m') F_h (x) conj F_h of lo_phonon_kernel,
    // numerics/reference/kernels.jl:321-356, and the tabulated kernels of
    // numerics/optimized/kernels.jl:303-320, compressed on the host).  Per
    // chunk of up to kSepChunk terms:
    //   stage 1 (term i, batch (c,d)):  Z_i[e + NE m + NE Nk (c,d)] =
    //            sum_m' radial_i[m + Nk m'] wk[m'] G[e + NE m' + NE Nk (c,d)]
    //   stage 2 (one GEMM over the chunk, K = (c,d,i)):
    //            S[(e,m), (a,b)] = alpha q sum_k Z[(e,m), k] block[(a,b), k] + beta S
    // The rows of stage 2 are the (e, m) pairs, contiguous in the E-fastest
    // layout, so S and Z are plain column-major (NE Nk) x N^2 matrices.
    for (int fi = 0; fi < fields; ++fi) {
    const int J = op.J;
    const long long Mr = NEl * Nk;                // stage-2 rows
    const size_t zfield = (size_t)Mr * N2;        // one intermediate field
    Cx<R>* Z = (Cx<R>*)work;
    const int jmax = J < kSepChunk ? J : kSepChunk;  // terms per chunk
    float* awork = (float*)((char*)work + (jmax * zfield * sizeof(Cx<R>) + kOperandAlign - 1) / kOperandAlign * kOperandAlign);
    // complex64 with tensor-core stage-1 operands: G split once for all chunks,
    // rows (e, (c,d)), K = m', behind the stage-2 work area
    float* gwork = awork + tc_a_work_floats2((int)Mr, jmax * N2);
    int s;
    if (sizeof(R) == 4 && op.tc_stage1 && (s = tc_split_rows(NE * N2, Nk, Gv[fi], NEl, NEl * Nk, gwork, st))) return s;
    for (int c = 0, i0 = 0; i0 < J; ++c, i0 += kSepChunk) {
      const int jc = min(kSepChunk, J - i0);
      if (sizeof(R) == 4 && op.tc_stage1) {
        // stage 1 on the tensor cores: rows (e, (c,d)), columns (m, i), K = m';
        // the output index (e, m, (c,d), i) is the chunk's intermediate layout
        if ((s = launch_tc_presplit(NE * N2, Nk * jc, Nk, op.tc_stage1[c], gwork, Z, NEl, Nk, N2, 1.0, 0.0,
                                    op.status, st)))
          return s;
      } else
      for (int i = i0; i < i0 + jc; ++i) {
        GemmArgs<R> g{};
        g.M = NE; g.Nout = Nk; g.K = Nk; g.batch = N2;
        g.A[0] = G[fi]; g.lda = NEl; g.a_b = Mr; g.wk = wk; g.wk_mod = Nk;
        g.B = (const Cx<R>*)op.radial + (size_t)Nk * Nk * i; g.ldb = Nk;
        g.C[0] = Z + zfield * (i - i0); g.ldc = NEl; g.c_b = Mr; g.bcast = 1;
        g.alpha = 1.0; g.beta = 0.0;
        if ((s = launch_gemm(g, st))) return s;
      }
      const double bc = c == 0 ? beta : 1.0;
      const Cx<R>* blk = (const Cx<R>*)op.block + (size_t)N2 * N2 * i0;
      const bool i8 = sizeof(R) == 8 && takes_i8(op, (int)Mr, 1, N2, jc * N2);
      if (i8) {
        const void* A[1] = {Z};
        void* C[1] = {Sv[fi]};
        if ((s = launch_i8_gemm((int)Mr, 1, N2, jc * N2, A, Mr, nullptr, 1, blk, N2, C, Mr, alpha_q, bc, op.i8_work,
                                op.i8_bytes, op.status, st)))
          return s;
      }
      if (op.tc_chunks) {
        if ((s = launch_tc_contraction2((int)Mr, N2, jc * N2, op.tc_chunks[c], Z, Sv[fi], alpha_q, bc, awork, op.status,
                                        st)))
          return s;
      } else {
        GemmArgs<R> f{};
        f.M = (int)Mr; f.Nout = N2; f.K = jc * N2; f.batch = 1;
        f.A[0] = Z; f.lda = Mr;
        f.B = blk; f.ldb = N2;
        f.C[0] = S[fi]; f.ldc = Mr; f.bcast = 1;
        f.alpha = alpha_q; f.beta = bc;
        if (i8) f.i8_level = (const int*)op.i8_work;
        if ((s = launch_gemm(f, st))) return s;
      }
    }
    }  // fields
    return QCL_OK;
  }
  set_last_error("unknown kernel operator kind %d", op.kind);
  return QCL_ARG;
}

// Stage-1 operand of a chunk of separable-sum terms [i0, i0 + jc):
// Mop[(m + Nk i') + Nk jc m'] = radial[m + Nk m' + Nk^2 (i0 + i')] (complex64).
__global__ void sep_radial_gather_kernel(int Nk, int i0, int jc, const Cx<float>* __restrict__ radial,
                                         Cx<float>* __restrict__ out) {
  const long long n = (long long)Nk * jc * Nk;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(t % Nk), ip = (int)((t / Nk) % jc), mp = (int)(t / ((long long)Nk * jc));
    out[t] = radial[(size_t)m + (size_t)Nk * mp + (size_t)Nk * Nk * (i0 + ip)];
  }
}

// Tensor-core operands of a complex64 separable sum: per chunk of kSepChunk
// terms the stage-2 operand (the stacked blocks, N^2 x jc N^2) and the
// stage-1 operand (the radial factors with the momentum weights, Nk jc x Nk).
int sep_build_tc_operands(int Nk, int N, int J, const void* radial_c64, const void* block_c64, const double* wk,
                          std::vector<void*>& stage2, std::vector<void*>& stage1, cudaStream_t st) {
  const int N2 = N * N;
  void* tmp = nullptr;
  QCL_CUDA_CHECK(cudaMalloc(&tmp, (size_t)Nk * Nk * kSepChunk * sizeof(Cx<float>)));
  int s = QCL_OK;
  for (int i0 = 0; i0 < J && !s; i0 += kSepChunk) {
    const int jc = J - i0 < kSepChunk ? J - i0 : kSepChunk;
    void* b = nullptr;
    s = tc_build_operator2(N2, jc * N2, 1, (const Cx<float>*)block_c64 + (size_t)N2 * N2 * i0, nullptr, &b, st);
    if (b) stage2.push_back(b);
    if (s) break;
    sep_radial_gather_kernel<<<grid_cap((long long)Nk * jc * Nk, 256), 256, 0, st>>>(
        Nk, i0, jc, (const Cx<float>*)radial_c64, (Cx<float>*)tmp);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      s = cuda_status(e, "sep_radial_gather_kernel");
      break;
    }
    b = nullptr;
    s = tc_build_operator2(Nk * jc, Nk, Nk, tmp, wk, &b, st);
    if (b) stage1.push_back(b);
    cudaStreamSynchronize(st);  // tmp is reused by the next chunk
  }
  cudaStreamSynchronize(st);
  cudaFree(tmp);
  return s;
}

size_t contraction_work_elems(const KernelOpDev& op, int NE, int Nk, int N) {
  if (op.kind == QCL_KERNEL_MOMENTUM_INDEPENDENT) return (size_t)NE * N * N;
  if (op.kind == QCL_KERNEL_DENSE && op.tc_bop) return (tc_a_work_floats(NE, Nk * N * N) + 1) / 2;  // complex64 units
  if (op.kind == QCL_KERNEL_IFR) return 2 * (size_t)NE * op.J * Nk;
  if (op.kind == QCL_KERNEL_LOW_RANK) return (size_t)NE * op.J;
  if (op.kind == QCL_KERNEL_SEPARABLE_SUM) {
    // kSepChunk intermediate fields (field precision), then for complex64
    // tensor-core chunks the stage-2 A operand (floats) in complex64 units
    const int jmax = op.J < kSepChunk ? op.J : kSepChunk;
    const size_t zf = (size_t)jmax * NE * Nk * N * N;
    if (op.tc_chunks)
      return zf + kOperandAlign / sizeof(Cx<float>) +
             (tc_a_work_floats2(NE * Nk, jmax * N * N) + (op.tc_stage1 ? tc_a_work_floats2(NE * N * N, Nk) : 0) + 1) / 2;
    return zf;
  }
  return 0;
}

// The area for the whole operands, or, for a stage-2 product of a separable
// sum with many more rows than columns, for a panel of rows.
size_t contraction_i8_bytes(const KernelOpDev& op, int NE, int Nk, int N, size_t* least) {
  const int N2 = N * N;
  if (least) *least = 0;
  if (op.kind == QCL_KERNEL_DENSE) {
    const int Nc = Nk * N2;
    if (!i8_worthwhile(NE, 2, Nc, Nc)) return 0;
    if (least) *least = i8_least_bytes(NE, 2, Nc, Nc);
    return i8_work_bytes(NE, 2, Nc, Nc);
  }
  if (op.kind == QCL_KERNEL_SEPARABLE_SUM) {
    const long long Mr = (long long)NE * Nk;
    const int K = (op.J < kSepChunk ? op.J : kSepChunk) * N2;
    if (!i8_worthwhile((int)Mr, 1, N2, K)) return 0;
    if (least) *least = i8_least_bytes((int)Mr, 1, N2, K);
    return i8_work_bytes((int)Mr, 1, N2, K, 4736);
  }
  return 0;
}

// The second field's scratch is as large as the first's; where it is not given
// (work2 == NULL), an operator's maps gain nothing, or the momenta of both
// fields exceed a grid's z extent, the fields go one by one.
int launch_contraction_pair(int precision, const KernelOpDev& op, int NE, int Nk, int N, const double* wk,
                            const void* const* G, void* const* S, double alpha_q, void* work, void* work2,
                            cudaStream_t st) {
  const bool scratch = op.kind != QCL_KERNEL_DENSE && op.kind != QCL_KERNEL_SEPARABLE_SUM;
  if (scratch && (!work2 || 2ll * Nk > 65535)) {
    for (int f = 0; f < 2; ++f)
      if (int s = launch_contraction(precision, op, NE, Nk, N, wk, G[f], S[f], alpha_q, 0.0, work, st)) return s;
    return QCL_OK;
  }
  if (precision == QCL_C128) return contraction_t<double>(op, NE, Nk, N, wk, 2, G, S, alpha_q, 0.0, work, work2, st);
  return contraction_t<float>(op, NE, Nk, N, wk, 2, G, S, alpha_q, 0.0, work, work2, st);
}

int launch_contraction(int precision, const KernelOpDev& op, int NE, int Nk, int N, const double* wk, const void* G,
                       void* S, double alpha_q, double beta, void* work, cudaStream_t st) {
  const void* Gv[1] = {G};
  void* Sv[1] = {S};
  if (precision == QCL_C128) return contraction_t<double>(op, NE, Nk, N, wk, 1, Gv, Sv, alpha_q, beta, work, nullptr, st);
  return contraction_t<float>(op, NE, Nk, N, wk, 1, Gv, Sv, alpha_q, beta, work, nullptr, st);
}

}  // namespace qcl
