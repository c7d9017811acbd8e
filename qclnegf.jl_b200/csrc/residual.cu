// Fixed-point residual suite, FP64.
//
// Reference: production_residual_suite (numerics/optimized/residuals.jl:
// 537-770) with the definitions of numerics/reference/validation.jl:33-103:
//   r_D   = max_em ||D G - I||_F / (||D||_F ||G||_F + sqrt(N))
//   r_A   = sqrt(sum ||A - G Gam G^H||^2) / (sqrt(sum ||A||^2) + 1e-14)
//   r_K   = sqrt(sum ||G< - G S^<_cand G^H||^2) / (sqrt(sum ||G<||^2) + 1e-14)
//   r_PSD = max over {A, -iG<, iG>, Gam, -i G S< G^H, i G S> G^H} of
//           max(0, -lmin - 64 n eps max(|l|max, 1)) / |l|max
//           (psd_error_budget, numerics/reference/positivity_diagnostics.jl:
//           15-40, witness ratio :60-90)
//   r_caus = max_em max(0, lmax(Im_H SR)) / (||SR||_2 + 1e-14)
// with D = eps I - h - SR_total, Gam = i(S>_total - S<_total), A = i(G - G^H).
//
// B200 mapping: one team per (E,k) block as in the Dyson kernel.  Only the
// extreme Hermitian eigenvalues enter the suite (LAPACK zheev in the
// reference, residuals.jl:311-353): each matrix is reduced to real
// tridiagonal form by team-parallel Householder steps, and Sturm counts on the
// tridiagonal settle the positive (causal) case with one count; lmin / lmax
// are found by multisection only for indefinite blocks.  The spectral norm of
// SR (zgesvd, :355-409) is lmax(SR SR^H), needed only when lmax(Im SR) > 0.
// The full spectrum (qcl_hermitian_eigvals) uses a team-parallel complex
// Jacobi iteration.  Per-block partial results go to global memory and are
// reduced in a fixed order.
#include <mutex>

#include "residual.cuh"

namespace qcl {

template <typename RS, int NP, int BPC>
__device__ __forceinline__ void load_tile(const Cx<RS>* X, Cx<double>* bufs, int e0, int m, int NE, int Nk, int N) {
  load_blocks<RS, double, NP, BPC>(X, bufs, (size_t)NP * NP, e0, m, NE, Nk, N);
}

template <typename RS, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT) residual_kernel(ResidualArgs<RS> p) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bG = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* bX = bG + BPC * MSZ;
  Cx<double>* bW = bX + BPC * MSZ;
  Cx<double>* bH = bW + BPC * MSZ;
  ResScratch<NP>* scr = reinterpret_cast<ResScratch<NP>*>(bH + BPC * MSZ);
  const int N = p.N, NE = p.NE, Nk = p.Nk;
  const int m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT;
  const int e = e0 + team;
  const bool live = e < NE;
  Cx<double>* G = bG + team * MSZ;
  Cx<double>* X = bX + team * MSZ;
  Cx<double>* W = bW + team * MSZ;
  Cx<double>* H = bH + team * MSZ;
  ResScratch<NP>& S = scr[team];
  const Cx<double> one = cx<double>(1, 0), mi = cx<double>(0, -1), pi = cx<double>(0, 1);

  if (p.part == RES_PART_RK) {  // launch-uniform
    // r_K alone: ||G< - G S<_cand G^H||^2 and ||G<||^2 of this block
    load_tile<RS, NP, BPC>(p.GR, bG, e0, m, NE, Nk, N);
    load_tile<RS, NP, BPC>(p.GL, bX, e0, m, NE, Nk, N);
    load_tile<RS, NP, BPC>(p.SLc, bW, e0, m, NE, Nk, N);
    __syncthreads();
    team_matmul<double, double, NP>(G, W, H, N, tt, false);  // H = G S<_cand
    team_sync<TT>(team);
    team_matmul<double, double, NP>(H, G, W, N, tt, true);   // W = H G^H
    team_sync<TT>(team);
    double kNum = 0, kDen = 0;
    tile_for<NP, TT>(N, tt, [&](int i, int j) {
      const Cx<double> a = X[sw<NP>(i, j)], q = W[sw<NP>(i, j)];
      kNum += (a.x - q.x) * (a.x - q.x) + (a.y - q.y) * (a.y - q.y);
      kDen += a.x * a.x + a.y * a.y;
    });
    team_sum2<TT>(kNum, kDen, tt, S.red, team);
    if (tt == 0 && live) {
      double* o = p.block_out + kResidualBlockDoubles * ((size_t)e + (size_t)NE * m);
      o[3] = isfinite(kNum) ? kNum : INFINITY;
      o[4] = isfinite(kDen) ? kDen : INFINITY;
    }
    return;
  }

  load_tile<RS, NP, BPC>(p.GR, bG, e0, m, NE, Nk, N);
  load_tile<RS, NP, BPC>(p.SR, bX, e0, m, NE, Nk, N);
  __syncthreads();
  const double eps_e = live ? p.eps[e] : 0.0;

  // ---- causality: lmax(Im_H SR) --------------------------------------------
  double caus_num = 0;
  {
    double bad = 0;
    tile_for<NP, TT>(N, tt, [&](int i, int j) {
      const Cx<double> a = X[sw<NP>(i, j)], b = X[sw<NP>(j, i)];
      if (!isfinite(a.x) || !isfinite(a.y)) bad = 1;
      // (a - conj(b)) / (2i)
      const double dx = a.x - b.x, dy = a.y + b.y;
      H[sw<NP>(i, j)] = cx<double>(0.5 * dy, -0.5 * dx);
    });
    bad = team_max<TT>(bad, tt, S.red, team);
    if (bad != 0) {
      caus_num = INFINITY;
    } else {
      // the causal case, -Im_H SR positive definite, is settled by one LDL^T
      tile_for<NP, TT>(N, tt, [&](int i, int j) {
        const Cx<double> v = H[sw<NP>(i, j)];
        W[sw<NP>(i, j)] = cx<double>(-v.x, -v.y);
      });
      team_sync<TT>(team);
      if (!team_posdef<NP, TT>(W, N, 0.0, tt, team)) caus_num = fmax(0.0, team_lmax<NP, TT>(H, N, tt, S, team, true));
      team_sync<TT>(team);
    }
  }
  double caus = 0;
  if (caus_num > 0 && isfinite(caus_num)) {  // team-uniform
    // ||SR||_2^2 = lmax(SR SR^H)
    team_matmul<double, double, NP>(X, X, H, N, tt, true);
    team_sync<TT>(team);
    const double lmax = team_lmax<NP, TT>(H, N, tt, S, team, false);
    caus = caus_num / (sqrt(fmax(lmax, 0.0)) + 1e-14);
  } else if (!isfinite(caus_num)) {
    caus = INFINITY;
  }

  // ---- r_D -------------------------------------------------------------------
  double nD = 0, nG = 0;
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> hv = p.h[(size_t)m + (size_t)Nk * ((size_t)i + (size_t)N * j)];
    Cx<double> d = X[sw<NP>(i, j)];
    d = cx<double>(-hv.x - d.x, -hv.y - d.y);
    if (i == j) d.x += eps_e;
    X[sw<NP>(i, j)] = d;
    nD += d.x * d.x + d.y * d.y;
    const Cx<double> g = G[sw<NP>(i, j)];
    nG += g.x * g.x + g.y * g.y;
  });
  team_sum2<TT>(nD, nG, tt, S.red, team);
  team_sync<TT>(team);
  team_matmul<double, double, NP>(X, G, W, N, tt, false);
  team_sync<TT>(team);
  double nR = 0;
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    Cx<double> v = W[sw<NP>(i, j)];
    if (i == j) v.x -= 1;
    nR += v.x * v.x + v.y * v.y;
  });
  nR = team_sum<TT>(nR, tt, S.red, team);
  double rD = sqrt(nR) / (sqrt(nD) * sqrt(nG) + sqrt((double)N));
  if (!isfinite(rD)) rD = INFINITY;

  // ---- spectral function A and its positivity ---------------------------------
  double psd = 0;
  // positivity witness of this block: the largest ratio over the six matrices,
  // the lowest kind index on ties (kinds: 0 spectral, 1 occupied, 2
  // unoccupied, 3 broadening, 4 raw occupied, 5 raw unoccupied); a
  // non-finite raw product is not a witness candidate
  double wr = -1.0, wk = -1.0;
  auto witness = [&](double r, int kind) {
    psd = fmax(psd, r);
    if (kind >= 4 && !isfinite(r)) return;
    if (r > wr || (r == wr && kind < wk)) {
      wr = r;
      wk = kind;
    }
  };
  // four tiles per team: G (G^R), X, W, H; X keeps A = i (G - G^H) (D is no
  // longer needed after r_D) until r_A is formed
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> g = G[sw<NP>(i, j)], gt = G[sw<NP>(j, i)];
    X[sw<NP>(i, j)] = pi * cx<double>(g.x - gt.x, g.y + gt.y);
  });
  team_sync<TT>(team);
  witness(psd_of<NP, TT>(X, one, H, N, tt, S, team), 0);

  // ---- Gamma = i (S> - S<), its positivity, r_A ---------------------------------
  __syncthreads();
  load_tile<RS, NP, BPC>(p.SG, bW, e0, m, NE, Nk, N);
  load_tile<RS, NP, BPC>(p.SL, bH, e0, m, NE, Nk, N);
  __syncthreads();
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> g = W[sw<NP>(i, j)], l = H[sw<NP>(i, j)];
    W[sw<NP>(i, j)] = pi * cx<double>(g.x - l.x, g.y - l.y);
  });
  team_sync<TT>(team);
  witness(psd_of<NP, TT>(W, one, H, N, tt, S, team), 3);
  team_matmul<double, double, NP>(G, W, H, N, tt, false);  // H = G Gam
  team_sync<TT>(team);
  team_matmul<double, double, NP>(H, G, W, N, tt, true);   // W = G Gam G^H
  team_sync<TT>(team);
  double aNum = 0, aDen = 0;
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> a = X[sw<NP>(i, j)], q = W[sw<NP>(i, j)];
    aNum += (a.x - q.x) * (a.x - q.x) + (a.y - q.y) * (a.y - q.y);
    aDen += a.x * a.x + a.y * a.y;
  });
  team_sum2<TT>(aNum, aDen, tt, S.red, team);

  // ---- raw Keldysh products -i G S< G^H, i G S> G^H ------------------------------
  for (int which = 0; which < 2; ++which) {
    __syncthreads();
    load_tile<RS, NP, BPC>(which == 0 ? p.SL : p.SG, bX, e0, m, NE, Nk, N);
    __syncthreads();
    team_matmul<double, double, NP>(G, X, W, N, tt, false);
    team_sync<TT>(team);
    team_matmul<double, double, NP>(W, G, X, N, tt, true);
    team_sync<TT>(team);
    witness(psd_of<NP, TT>(X, which == 0 ? mi : pi, H, N, tt, S, team), 4 + which);
  }

  // ---- G< : positivity and r_K against the candidate lesser self-energy ----------
  __syncthreads();
  const bool with_rk = p.part == RES_PART_ALL;  // launch-uniform
  load_tile<RS, NP, BPC>(p.GL, bX, e0, m, NE, Nk, N);
  if (with_rk) load_tile<RS, NP, BPC>(p.SLc, bW, e0, m, NE, Nk, N);
  __syncthreads();
  witness(psd_of<NP, TT>(X, mi, H, N, tt, S, team), 1);
  double kNum = 0, kDen = 0;
  if (with_rk) {
    team_matmul<double, double, NP>(G, W, H, N, tt, false);
    team_sync<TT>(team);
    team_matmul<double, double, NP>(H, G, W, N, tt, true);
    team_sync<TT>(team);
    tile_for<NP, TT>(N, tt, [&](int i, int j) {
      const Cx<double> a = X[sw<NP>(i, j)], q = W[sw<NP>(i, j)];
      kNum += (a.x - q.x) * (a.x - q.x) + (a.y - q.y) * (a.y - q.y);
      kDen += a.x * a.x + a.y * a.y;
    });
    team_sum2<TT>(kNum, kDen, tt, S.red, team);
  }

  // ---- G> positivity ---------------------------------------------------------------
  __syncthreads();
  load_tile<RS, NP, BPC>(p.GG, bX, e0, m, NE, Nk, N);
  __syncthreads();
  witness(psd_of<NP, TT>(X, pi, H, N, tt, S, team), 2);

  if (tt == 0 && live) {
    double* o = p.block_out + kResidualBlockDoubles * ((size_t)e + (size_t)NE * m);
    o[0] = rD;
    o[1] = isfinite(aNum) ? aNum : INFINITY;
    o[2] = isfinite(aDen) ? aDen : INFINITY;
    if (with_rk) {
      o[3] = isfinite(kNum) ? kNum : INFINITY;
      o[4] = isfinite(kDen) ? kDen : INFINITY;
    }
    o[5] = psd;
    o[6] = caus;
    o[7] = wr;
    o[8] = wk;
  }
}

template <typename RS, int NP, int BPC> static int launch_residual_t(const ResidualArgs<RS>& a, cudaStream_t st) {
  constexpr int TT = Tile<NP>::TT;
  // four tiles per team (G, X, W, H) and the scratch
  constexpr size_t smem = 4 * (size_t)BPC * NP * NP * sizeof(Cx<double>) + BPC * sizeof(ResScratch<NP>);
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(residual_kernel<RS, NP, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  dim3 grid((a.NE + BPC - 1) / BPC, a.Nk);
  residual_kernel<RS, NP, BPC><<<grid, BPC * TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("residual_kernel");
  return QCL_OK;
}

template <typename RS> static int launch_residual_p(const ResidualArgs<RS>& a, cudaStream_t st) {
  switch (padded_size(a.N)) {
    case 8:
    case 16: return launch_residual_rows_small(a, st);
    case 24:
    case 32: return launch_residual_rows_large(a, st);
    case 48: return launch_residual_t<RS, 48, 1>(a, st);
    default:
      set_last_error("basis size N_b=%d exceeds the supported maximum 48", a.N);
      return QCL_UNSUPPORTED;
  }
}

// Batched Hermitian eigenvalues: matrices (n x n, column-major, complex128)
// stored back to back; one team per matrix.
template <int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT) eigvals_kernel(int n, long long count,
                                                                    const Cx<double>* __restrict__ A, double* vals) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bH = reinterpret_cast<Cx<double>*>(smem_raw);
  ResScratch<NP>* scr = reinterpret_cast<ResScratch<NP>*>(bH + BPC * MSZ);
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT;
  const long long mat = (long long)blockIdx.x * BPC + team;
  const bool live = mat < count;
  Cx<double>* H = bH + team * MSZ;
  for (int idx = tt; idx < n * n; idx += TT) {
    const int i = idx % n, j = idx / n;
    H[sw<NP>(i, j)] = live ? A[(size_t)mat * n * n + idx] : cx<double>(i == j ? 1.0 : 0.0, 0.0);
  }
  team_sync<TT>(team);
  // Hermitian part (as zheev reads one triangle of a Hermitian input)
  for (int idx = tt; idx < n * n; idx += TT) {
    const int i = idx % n, j = idx / n;
    if (i > j) {
      const Cx<double> a = H[sw<NP>(i, j)], b = H[sw<NP>(j, i)];
      const Cx<double> m = cx<double>(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
      H[sw<NP>(i, j)] = m;
      H[sw<NP>(j, i)] = conj(m);
    } else if (i == j) {
      H[sw<NP>(i, i)] = cx<double>(H[sw<NP>(i, i)].x, 0.0);
    }
  }
  team_sync<TT>(team);
  team_eigvals<NP, TT>(H, n, tt, scr[team], team);
  if (live)
    for (int i = tt; i < n; i += TT) vals[(size_t)mat * n + i] = scr[team].vals[i];
}

int launch_eigvals(int n, long long count, const void* A, double* vals, cudaStream_t st) {
  const int NP = padded_size(n);
  if (NP == 0) {
    set_last_error("matrix size %d exceeds the supported maximum 48", n);
    return QCL_UNSUPPORTED;
  }
#define EIGV(NPV, BPCV)                                                                                       \
  do {                                                                                                         \
    constexpr size_t smem = (size_t)BPCV * NPV * NPV * sizeof(Cx<double>) + BPCV * sizeof(ResScratch<NPV>);  \
    cudaFuncSetAttribute(eigvals_kernel<NPV, BPCV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    eigvals_kernel<NPV, BPCV><<<(unsigned)((count + BPCV - 1) / BPCV), BPCV * Tile<NPV>::TT, smem, st>>>(    \
        n, count, (const Cx<double>*)A, vals);                                                                \
  } while (0)
  switch (NP) {
    case 8: EIGV(8, 8); break;
    case 16: EIGV(16, 4); break;
    case 24: EIGV(24, 4); break;
    case 32: EIGV(32, 2); break;
    default: EIGV(48, 1); break;
  }
#undef EIGV
  QCL_LAUNCH_CHECK("eigvals_kernel");
  return QCL_OK;
}

// ---------------------------------------------------------------------------
// Condition number and Dyson scale per (E,k) block: the condition_number and
// dyson_scale fields of GreenState (domain/types.jl:733-740) as
// retarded_green / _retarded_green_production write them
// (numerics/reference/greens.jl:30-41, production_operators.jl:1362-1380):
//   D = (eps_e + i eta) I - h_m - SigmaR_em,  s = max_a sum_b |D_ab|,
//   kappa = cond_2(D) = ||D||_2 ||D^-1||_2.
// D is rebuilt from the Dyson inputs and D^-1 is the G^R the Dyson kernel
// produced for them.  The reference takes cond(D) from an SVD (zgesvd); here
// each spectral norm is sqrt(lmax(X X^H)) by the tridiagonal multisection of
// the residual suite.  Nothing in the SCBA loop reads kappa, so it is computed
// on request only.
// ---------------------------------------------------------------------------
template <typename RS> struct CondArgs {
  int NE, Nk, N;
  const double* eps;
  double eta;
  const Cx<double>* h;
  const Cx<RS>* SR;  // may be NULL (Sigma^R = 0)
  const Cx<RS>* GR;
  double* kappa;     // (N_E, N_k) or NULL
  double* scale;     // (N_E, N_k) or NULL
};

template <typename RS, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT) condition_kernel(CondArgs<RS> p) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bG = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* bX = bG + BPC * MSZ;
  Cx<double>* bH = bX + BPC * MSZ;
  ResScratch<NP>* scr = reinterpret_cast<ResScratch<NP>*>(bH + BPC * MSZ);
  const int N = p.N, NE = p.NE, Nk = p.Nk;
  const int m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT;
  const int e = e0 + team;
  const bool live = e < NE;
  Cx<double>* G = bG + team * MSZ;
  Cx<double>* X = bX + team * MSZ;
  Cx<double>* H = bH + team * MSZ;
  ResScratch<NP>& S = scr[team];

  load_tile<RS, NP, BPC>(p.GR, bG, e0, m, NE, Nk, N);
  if (p.SR) load_tile<RS, NP, BPC>(p.SR, bX, e0, m, NE, Nk, N);
  __syncthreads();
  const double eps_e = live ? p.eps[e] : 0.0;
  for (int idx = tt; idx < N * N; idx += TT) {
    const int i = idx % N, j = idx / N;
    const Cx<double> hv = p.h[(size_t)m + (size_t)Nk * ((size_t)i + (size_t)N * j)];
    const Cx<double> sr = p.SR ? X[sw<NP>(i, j)] : cx<double>(0, 0);
    Cx<double> d = cx<double>(-hv.x - sr.x, -hv.y - sr.y);
    if (i == j) {
      d.x += eps_e;
      d.y += p.eta;
    }
    X[sw<NP>(i, j)] = d;
  }
  team_sync<TT>(team);
  // s = max row sum |D_ab| (row a per thread, then a team max)
  double rowmax = 0;
  for (int a = tt; a < N; a += TT) {
    double r = 0;
    for (int b = 0; b < N; ++b) {
      const Cx<double> d = X[sw<NP>(a, b)];
      r += hypot(d.x, d.y);
    }
    rowmax = fmax(rowmax, r);
  }
  rowmax = team_max<TT>(rowmax, tt, S.red, team);
  double kappa = 0;
  if (p.kappa) {
    team_matmul<double, double, NP>(X, X, H, N, tt, true);  // D D^H
    team_sync<TT>(team);
    const double lD = team_lmax<NP, TT>(H, N, tt, S, team, false);
    team_sync<TT>(team);
    team_matmul<double, double, NP>(G, G, H, N, tt, true);  // D^-1 D^-H
    team_sync<TT>(team);
    const double lG = team_lmax<NP, TT>(H, N, tt, S, team, false);
    kappa = (isfinite(lD) && isfinite(lG)) ? sqrt(fmax(lD, 0.0)) * sqrt(fmax(lG, 0.0)) : INFINITY;
  }
  if (live && tt == 0) {
    const size_t o = (size_t)e + (size_t)NE * m;
    if (p.kappa) p.kappa[o] = kappa;
    if (p.scale) p.scale[o] = rowmax;
  }
}

template <typename RS, int NP, int BPC> static int launch_condition_t(const CondArgs<RS>& a, cudaStream_t st) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t smem = 3 * (size_t)BPC * NP * NP * sizeof(Cx<double>) + BPC * sizeof(ResScratch<NP>);
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(condition_kernel<RS, NP, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  dim3 grid((a.NE + BPC - 1) / BPC, a.Nk);
  condition_kernel<RS, NP, BPC><<<grid, BPC * TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("condition_kernel");
  return QCL_OK;
}

template <typename RS> static int launch_condition_p(const CondArgs<RS>& a, cudaStream_t st) {
  switch (padded_size(a.N)) {
    case 8: return launch_condition_t<RS, 8, 8>(a, st);
    case 16: return launch_condition_t<RS, 16, 4>(a, st);
    case 24: return launch_condition_t<RS, 24, 4>(a, st);
    case 32: return launch_condition_t<RS, 32, 2>(a, st);
    case 48: return launch_condition_t<RS, 48, 1>(a, st);
    default:
      set_last_error("basis size N_b=%d exceeds the supported maximum 48", a.N);
      return QCL_UNSUPPORTED;
  }
}

int launch_condition(int precision, int NE, int Nk, int N, const double* eps, double eta, const void* h,
                     const void* SR, const void* GR, double* kappa, double* scale, cudaStream_t st) {
  if (precision == QCL_C128) {
    CondArgs<double> a{NE, Nk, N, eps, eta, (const Cx<double>*)h, (const Cx<double>*)SR, (const Cx<double>*)GR,
                       kappa, scale};
    return launch_condition_p<double>(a, st);
  }
  CondArgs<float> a{NE, Nk, N, eps, eta, (const Cx<double>*)h, (const Cx<float>*)SR, (const Cx<float>*)GR, kappa,
                    scale};
  return launch_condition_p<float>(a, st);
}

// A = i (G^R - G^R^H) per block (spectral_function, numerics/reference/
// greens.jl:50-57; the A field written by _green_state_production,
// production_operators.jl:1387-1415).  One thread per element; the transposed
// partner is read from the same (E,k) column, so both reads stay coalesced
// along E.
template <typename R>
__global__ void spectral_kernel(int NE, int Nk, int N, const Cx<R>* __restrict__ GR, Cx<R>* __restrict__ A) {
  const long long blocks = (long long)NE * Nk, n = blocks * N * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long em = i % blocks, ab = i / blocks;
    const int a = (int)(ab % N), b = (int)(ab / N);
    const Cx<R> g = GR[i], gt = GR[em + blocks * ((long long)b + (long long)N * a)];
    const double dx = (double)g.x - (double)gt.x, dy = (double)g.y + (double)gt.y;  // G - G^H
    A[i] = cx<R>((R)(-dy), (R)dx);                                                  // i (G - G^H)
  }
}

int launch_spectral(int precision, int NE, int Nk, int N, const void* GR, void* A, cudaStream_t st) {
  const long long n = (long long)NE * Nk * N * N;
  long long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  if (g < 1) g = 1;
  if (precision == QCL_C128)
    spectral_kernel<double><<<(unsigned)g, 256, 0, st>>>(NE, Nk, N, (const Cx<double>*)GR, (Cx<double>*)A);
  else
    spectral_kernel<float><<<(unsigned)g, 256, 0, st>>>(NE, Nk, N, (const Cx<float>*)GR, (Cx<float>*)A);
  QCL_LAUNCH_CHECK("spectral_kernel");
  return QCL_OK;
}

// ---------------------------------------------------------------------------
// Positivity witness of the residual suite (_positivity_witness,
// numerics/reference/positivity_diagnostics.jl:41-91, collected per chunk in
// production_residual_suite, numerics/optimized/residuals.jl:662-726, and
// reduced by _production_positivity_witness, :773-779).  The reference scans
// the blocks in the order lin = m + N_k e (e slow, m fast; residuals.jl:
// 126-131) and the six matrices in kind order, keeping the first strict
// maximum of the ratio: the witness is the (block, kind) of largest ratio,
// lowest lin and then lowest kind on ties.  The residual kernel leaves each
// block's best (ratio, kind); a deterministic arg-max over the blocks picks
// the witness block, and one CTA recomputes that block's matrix and its full
// spectrum for the reported numbers.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool witness_better(double r, long long lin, double r2, long long lin2) {
  return r > r2 || (r == r2 && lin < lin2);
}

__global__ void witness_reduce_kernel(long long blocks, int NE, int Nk, const double* __restrict__ bo, double* partial) {
  double br = -2.0, bk = -1.0;
  long long bl = 0x7fffffffffffffffll;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < blocks;
       i += (long long)gridDim.x * blockDim.x) {
    const double* o = bo + kResidualBlockDoubles * i;
    const double r = isnan(o[7]) ? INFINITY : o[7];
    const long long lin = i / NE + (long long)Nk * (i % NE);
    if (witness_better(r, lin, br, bl)) {
      br = r;
      bl = lin;
      bk = o[8];
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double r2 = __shfl_xor_sync(0xffffffffu, br, off);
    const long long l2 = __shfl_xor_sync(0xffffffffu, bl, off);
    const double k2 = __shfl_xor_sync(0xffffffffu, bk, off);
    if (witness_better(r2, l2, br, bl)) {
      br = r2;
      bl = l2;
      bk = k2;
    }
  }
  __shared__ double sr[32], sk[32];
  __shared__ long long sl[32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sr[w] = br;
    sl[w] = bl;
    sk[w] = bk;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q)
      if (witness_better(sr[q], sl[q], br, bl)) {
        br = sr[q];
        bl = sl[q];
        bk = sk[q];
      }
    partial[3 * blockIdx.x + 0] = br;
    partial[3 * blockIdx.x + 1] = (double)bl;
    partial[3 * blockIdx.x + 2] = bk;
  }
}

template <typename RS> struct WitnessArgs {
  int NE, Nk, N, ncta;
  const Cx<RS>* GR;
  const Cx<RS>* GL;
  const Cx<RS>* GG;
  const Cx<RS>* SL;  // totals
  const Cx<RS>* SG;
  const double* partial;  // ncta x (ratio, lin, kind)
  double* out;            // kind, e, m, then the nine witness numbers
};

template <typename RS, int NP>
__global__ void __launch_bounds__(Tile<NP>::TT) witness_detail_kernel(WitnessArgs<RS> p) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* G = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* X = G + MSZ;
  Cx<double>* Y = X + MSZ;
  Cx<double>* H = Y + MSZ;
  ResScratch<NP>& S = *reinterpret_cast<ResScratch<NP>*>(H + MSZ);
  __shared__ double best[3];
  const int tt = threadIdx.x, N = p.N;
  if (tt == 0) {
    double br = -2.0, bk = -1.0;
    long long bl = 0x7fffffffffffffffll;
    for (int c = 0; c < p.ncta; ++c) {
      const double r = p.partial[3 * c];
      const long long l = (long long)p.partial[3 * c + 1];
      if (witness_better(r, l, br, bl)) {
        br = r;
        bl = l;
        bk = p.partial[3 * c + 2];
      }
    }
    best[0] = br;
    best[1] = (double)bl;
    best[2] = bk;
  }
  __syncthreads();
  const int kind = (int)best[2];
  if (kind < 0) {  // no block: the empty witness (positivity_diagnostics.jl:58-59)
    if (tt == 0) {
      const double v[12] = {-1, 0, 0, 0.0, 0.0, 0.0, -1.0, 0.0, 0.0, 0.0, 0.0, 1.0};
      for (int i = 0; i < 12; ++i) p.out[i] = v[i];
    }
    return;
  }
  const long long lin = (long long)best[1];
  const int e = (int)(lin / p.Nk), m = (int)(lin % p.Nk);
  load_tile<RS, NP, 1>(p.GR, G, e, m, p.NE, p.Nk, N);
  if (kind == 1) load_tile<RS, NP, 1>(p.GL, X, e, m, p.NE, p.Nk, N);
  if (kind == 2) load_tile<RS, NP, 1>(p.GG, X, e, m, p.NE, p.Nk, N);
  if (kind == 3 || kind == 4) load_tile<RS, NP, 1>(p.SL, Y, e, m, p.NE, p.Nk, N);
  if (kind == 3) load_tile<RS, NP, 1>(p.SG, X, e, m, p.NE, p.Nk, N);
  if (kind == 5) load_tile<RS, NP, 1>(p.SG, Y, e, m, p.NE, p.Nk, N);
  __syncthreads();
  const Cx<double> pi = cx<double>(0, 1);
  if (kind == 0 || kind == 3) {
    for (int idx = tt; idx < N * N; idx += TT) {
      const int i = idx % N, j = idx / N;
      Cx<double> v;
      if (kind == 0) {
        const Cx<double> g = G[sw<NP>(i, j)], gt = G[sw<NP>(j, i)];
        v = pi * cx<double>(g.x - gt.x, g.y + gt.y);  // A = i (G - G^H)
      } else {
        const Cx<double> g = X[sw<NP>(i, j)], l = Y[sw<NP>(i, j)];
        v = pi * cx<double>(g.x - l.x, g.y - l.y);  // Gam = i (S> - S<)
      }
      H[sw<NP>(i, j)] = v;
    }
    __syncthreads();
    for (int idx = tt; idx < N * N; idx += TT) X[sw<NP>(idx % N, idx / N)] = H[sw<NP>(idx % N, idx / N)];
  } else if (kind >= 4) {
    team_matmul<double, double, NP>(G, Y, H, N, tt, false);  // G S
    __syncthreads();
    team_matmul<double, double, NP>(H, G, X, N, tt, true);   // G S G^H
  }
  __syncthreads();
  const Cx<double> f = (kind == 1 || kind == 4) ? cx<double>(0, -1) : (kind == 2 || kind == 5) ? pi : cx<double>(1, 0);
  double bad = 0, herm = 0;
  for (int idx = tt; idx < N * N; idx += TT) {
    const int i = idx % N, j = idx / N;
    const Cx<double> v = f * X[sw<NP>(i, j)], u = f * X[sw<NP>(j, i)];
    if (!isfinite(v.x) || !isfinite(v.y)) bad = 1;
    H[sw<NP>(i, j)] = cx<double>(0.5 * (v.x + u.x), 0.5 * (v.y - u.y));
    const double dx = v.x - u.x, dy = v.y + u.y;  // v - conj(u)
    herm += dx * dx + dy * dy;
  }
  bad = team_max<TT>(bad, tt, S.red, 0);
  herm = team_sum<TT>(herm, tt, S.red, 0);
  if (bad != 0) {  // _nonfinite_positivity_witness (positivity_diagnostics.jl:56-57)
    if (tt == 0) {
      const double v[12] = {(double)kind, (double)e, (double)m, NAN, INFINITY, 1e-14, INFINITY, NAN, NAN, 1e-14, 0.0,
                            1.0};
      for (int i = 0; i < 12; ++i) p.out[i] = v[i];
    }
    return;
  }
  team_eigvals<NP, TT>(H, N, tt, S, 0);
  if (tt == 0) {
    double lmin = INFINITY, bn = 0;
    bool fin = true;
    for (int i = 0; i < N; ++i) {
      const double l = S.vals[i];
      fin = fin && isfinite(l);
      lmin = fmin(lmin, l);
      bn = fmax(bn, fabs(l));
    }
    double* o = p.out;
    o[0] = kind;
    o[1] = e;
    o[2] = m;
    if (!fin) {
      const double v[9] = {NAN, INFINITY, 1e-14, INFINITY, NAN, NAN, 1e-14, 0.0, 1.0};
      for (int i = 0; i < 9; ++i) o[3 + i] = v[i];
      return;
    }
    const double budget = 64.0 * N * 2.220446049250313e-16 * fmax(bn, 1.0);
    const double absolute = fmax(0.0, -lmin), den = fmax(bn, 2.2250738585072014e-308);
    o[3] = lmin;
    o[4] = bn;
    o[5] = budget;
    o[6] = fmax(0.0, absolute - budget) / den;
    o[7] = absolute;
    o[8] = absolute / den;
    o[9] = budget;
    o[10] = sqrt(herm) / 2;
    o[11] = 1.0;
  }
}

template <typename RS, int NP> static int launch_witness_detail_t(const WitnessArgs<RS>& a, cudaStream_t st) {
  constexpr size_t smem = 4 * (size_t)NP * NP * sizeof(Cx<double>) + sizeof(ResScratch<NP>);
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(witness_detail_kernel<RS, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  witness_detail_kernel<RS, NP><<<1, Tile<NP>::TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("witness_detail_kernel");
  return QCL_OK;
}

template <typename RS> static int launch_witness_detail_p(const WitnessArgs<RS>& a, cudaStream_t st) {
  switch (padded_size(a.N)) {
    case 8: return launch_witness_detail_t<RS, 8>(a, st);
    case 16: return launch_witness_detail_t<RS, 16>(a, st);
    case 24: return launch_witness_detail_t<RS, 24>(a, st);
    case 32: return launch_witness_detail_t<RS, 32>(a, st);
    case 48: return launch_witness_detail_t<RS, 48>(a, st);
    default:
      set_last_error("basis size N_b=%d exceeds the supported maximum 48", a.N);
      return QCL_UNSUPPORTED;
  }
}

// ---------------------------------------------------------------------------
// Causality / Keldysh guard of an Anderson-mixed state
// (_anderson_block_failure!, numerics/optimized/production_mixing.jl:48-96),
// per block of every family, n = N_b:
//   1  a non-finite entry in Sigma^R, Sigma< or Sigma>;
//   2  lmax(Im_H Sigma^R) > 64 eps max(||Sigma^R||_2, floatmin);
//   3  ||fX - (fX)^H||_F / 2 > b(X), 4  lmin(Herm fX) < -b(X), for (X, f) =
//      (Sigma<, -i), (Sigma>, i), b(X) = 64 n eps max(||X||_2, 1);
//   5  ||Sigma^R - Sigma^R^H - (Sigma> - Sigma<)||_F > 64 n eps max(||Sigma^R||_2,
//      ||Sigma<||_2, ||Sigma>||_2, 1).
// Every test first tries a sufficient condition that needs no spectrum:
// LDL^T certificates for the sign tests, and max |entry| <= ||X||_2 for the
// budgets; the exact spectral norms and extreme eigenvalues (tridiagonal
// multisection) are computed only for blocks those do not settle.  The first
// failing block in the reference's order (family, e, m; m fastest) is kept
// with its code by one atomicMin on (index << 3 | code).
// ---------------------------------------------------------------------------
constexpr int kGuardMaxFamilies = kMaxMixFields / 3;
template <typename RS> struct GuardArgs {
  int NE, Nk, N, nfam, pass;
  double eps;  // unit roundoff the budgets are scaled to (see launch_anderson_guard)
  const Cx<RS>* f[3 * kGuardMaxFamilies];
  AndersonMeta* meta;
};

template <int NP, int TT>
__device__ double team_maxabs(const Cx<double>* X, int N, int tt, ResScratch<NP>& S, int team) {
  double a = 0;
  for (int idx = tt; idx < N * N; idx += TT) {
    const Cx<double> v = X[sw<NP>(idx % N, idx / N)];
    a = fmax(a, hypot(v.x, v.y));
  }
  return team_max<TT>(a, tt, S.red, team);
}

// ||X||_2 = sqrt(lmax(X X^H)); W is scratch.
template <int NP, int TT>
__device__ double team_norm2(const Cx<double>* X, Cx<double>* W, int N, int tt, ResScratch<NP>& S, int team) {
  team_matmul<double, double, NP>(X, X, W, N, tt, true);
  team_sync<TT>(team);
  return sqrt(fmax(team_lmax<NP, TT>(W, N, tt, S, team, false), 0.0));
}

template <typename RS, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT) anderson_guard_kernel(GuardArgs<RS> p) {
  if (p.pass == 1 && !p.meta->fallback) return;
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  // the budgets of the reference (64 n eps ||X||, production_mixing.jl:48-118)
  // scaled to the rounding the checked fields actually carry
  const double eps = p.eps;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bR = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* bL = bR + BPC * MSZ;
  Cx<double>* bG = bL + BPC * MSZ;
  Cx<double>* bH = bG + BPC * MSZ;
  Cx<double>* bW = bH + BPC * MSZ;
  ResScratch<NP>* scr = reinterpret_cast<ResScratch<NP>*>(bW + BPC * MSZ);
  const int N = p.N, NE = p.NE, Nk = p.Nk, fam = blockIdx.z;
  const int m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT;
  const int e = e0 + team;
  const bool live = e < NE;
  Cx<double>* R = bR + team * MSZ;
  Cx<double>* L = bL + team * MSZ;
  Cx<double>* G = bG + team * MSZ;
  Cx<double>* H = bH + team * MSZ;
  Cx<double>* W = bW + team * MSZ;
  ResScratch<NP>& S = scr[team];
  load_tile<RS, NP, BPC>(p.f[3 * fam + 0], bR, e0, m, NE, Nk, N);
  load_tile<RS, NP, BPC>(p.f[3 * fam + 1], bL, e0, m, NE, Nk, N);
  load_tile<RS, NP, BPC>(p.f[3 * fam + 2], bG, e0, m, NE, Nk, N);
  __syncthreads();
  int code = 0;
  // finiteness of the three blocks (code 1; the reference tests Sigma^R first)
  double badR = 0, badLG = 0;
  for (int idx = tt; idx < N * N; idx += TT) {
    const int i = idx % N, j = idx / N;
    const Cx<double> r = R[sw<NP>(i, j)], l = L[sw<NP>(i, j)], g = G[sw<NP>(i, j)];
    if (!isfinite(r.x) || !isfinite(r.y)) badR = 1;
    if (!isfinite(l.x) || !isfinite(l.y) || !isfinite(g.x) || !isfinite(g.y)) badLG = 1;
  }
  badR = team_max<TT>(badR, tt, S.red, team);
  badLG = team_max<TT>(badLG, tt, S.red, team);
  double nR = -1;  // ||Sigma^R||_2 once computed
  if (badR != 0) code = 1;
  if (!code) {  // code 2: causality of Sigma^R
    for (int idx = tt; idx < N * N; idx += TT) {
      const int i = idx % N, j = idx / N;
      const Cx<double> a = R[sw<NP>(i, j)], b = R[sw<NP>(j, i)];
      // -(a - conj b) / (2i) = -Im_H
      W[sw<NP>(i, j)] = cx<double>(-0.5 * (a.y + b.y), 0.5 * (a.x - b.x));
    }
    team_sync<TT>(team);
    if (!team_posdef<NP, TT>(W, N, 0.0, tt, team)) {
      team_sync<TT>(team);
      for (int idx = tt; idx < N * N; idx += TT) {
        const int i = idx % N, j = idx / N;
        const Cx<double> a = R[sw<NP>(i, j)], b = R[sw<NP>(j, i)];
        H[sw<NP>(i, j)] = cx<double>(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));  // Im_H
      }
      team_sync<TT>(team);
      const double lmax = team_lmax<NP, TT>(H, N, tt, S, team, false);
      team_sync<TT>(team);
      nR = team_norm2<NP, TT>(R, W, N, tt, S, team);
      if (!(lmax <= 64 * eps * fmax(nR, 2.2250738585072014e-308))) code = 2;
    }
    team_sync<TT>(team);
  }
  if (!code && badLG != 0) code = 1;
  for (int which = 0; which < 2 && !code; ++which) {  // codes 3, 4
    const Cx<double>* X = which == 0 ? L : G;
    const double fs = which == 0 ? -1.0 : 1.0;  // f = fs * i
    double dF2 = 0, amax = 0;
    for (int idx = tt; idx < N * N; idx += TT) {
      const int i = idx % N, j = idx / N;
      const Cx<double> a = X[sw<NP>(i, j)], b = X[sw<NP>(j, i)];
      const Cx<double> v = cx<double>(-fs * a.y, fs * a.x), u = cx<double>(-fs * b.y, fs * b.x);
      H[sw<NP>(i, j)] = cx<double>(0.5 * (v.x + u.x), 0.5 * (v.y - u.y));
      const double dx = v.x - u.x, dy = v.y + u.y;
      dF2 += dx * dx + dy * dy;
      amax = fmax(amax, hypot(a.x, a.y));
    }
    dF2 = team_sum<TT>(dF2, tt, S.red, team);
    amax = team_max<TT>(amax, tt, S.red, team);
    const double herm = sqrt(dF2) / 2;
    const double blo = 64.0 * N * eps * fmax(amax, 1.0);  // amax <= ||X||_2
    team_sync<TT>(team);
    if (herm <= blo && team_posdef<NP, TT>(H, N, blo, tt, team)) continue;
    team_sync<TT>(team);
    const double budget = 64.0 * N * eps * fmax(team_norm2<NP, TT>(X, W, N, tt, S, team), 1.0);
    team_sync<TT>(team);
    if (!(herm <= budget)) {
      code = 3;
      break;
    }
    for (int idx = tt; idx < N * N; idx += TT) {
      const int i = idx % N, j = idx / N;
      const Cx<double> a = X[sw<NP>(i, j)], b = X[sw<NP>(j, i)];
      const Cx<double> v = cx<double>(-fs * a.y, fs * a.x), u = cx<double>(-fs * b.y, fs * b.x);
      H[sw<NP>(i, j)] = cx<double>(0.5 * (v.x + u.x), 0.5 * (v.y - u.y));
    }
    team_sync<TT>(team);
    team_tridiagonalize<NP, TT>(H, N, tt, S, team);
    double lmin = INFINITY;
    bool fin = true;
    for (int i = 0; i < N; ++i) fin = fin && isfinite(S.d[i]) && (i + 1 >= N || isfinite(S.e2[i]));
    if (fin) lmin = tri_eig(S.d, S.e2, N, 1);
    team_sync<TT>(team);
    if (!(lmin >= -budget)) code = 4;
  }
  if (!code) {  // code 5: Keldysh identity
    double dF2 = 0, amax = 0;
    for (int idx = tt; idx < N * N; idx += TT) {
      const int i = idx % N, j = idx / N;
      const Cx<double> a = R[sw<NP>(i, j)], b = R[sw<NP>(j, i)], l = L[sw<NP>(i, j)], g = G[sw<NP>(i, j)];
      const double dx = (a.x - b.x) - (g.x - l.x), dy = (a.y + b.y) - (g.y - l.y);
      dF2 += dx * dx + dy * dy;
      amax = fmax(amax, fmax(hypot(a.x, a.y), fmax(hypot(l.x, l.y), hypot(g.x, g.y))));
    }
    dF2 = team_sum<TT>(dF2, tt, S.red, team);
    amax = team_max<TT>(amax, tt, S.red, team);
    const double dF = sqrt(dF2);
    if (!(dF <= 64.0 * N * eps * fmax(amax, 1.0))) {
      team_sync<TT>(team);
      if (nR < 0) nR = team_norm2<NP, TT>(R, W, N, tt, S, team);
      team_sync<TT>(team);
      const double nL = team_norm2<NP, TT>(L, W, N, tt, S, team);
      team_sync<TT>(team);
      const double nG = team_norm2<NP, TT>(G, W, N, tt, S, team);
      if (!(dF <= 64.0 * N * eps * fmax(fmax(nR, fmax(nL, nG)), 1.0))) code = 5;
    }
  }
  if (code && live && tt == 0) {
    const unsigned long long idx = (unsigned long long)fam * NE * Nk + (unsigned long long)e * Nk + m + 1;
    atomicMin(&p.meta->guard_key, (idx << 3) | (unsigned long long)code);
  }
}

template <typename RS, int NP, int BPC> static int launch_guard_t(const GuardArgs<RS>& a, cudaStream_t st) {
  constexpr int TT = Tile<NP>::TT;
  // five tiles per team (R, L, G, H, W) and the scratch
  constexpr size_t smem = 5 * (size_t)BPC * NP * NP * sizeof(Cx<double>) + BPC * sizeof(ResScratch<NP>);
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(anderson_guard_kernel<RS, NP, BPC>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured = true;
  }
  dim3 grid((a.NE + BPC - 1) / BPC, a.Nk, a.nfam);
  anderson_guard_kernel<RS, NP, BPC><<<grid, BPC * TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("anderson_guard_kernel");
  return QCL_OK;
}

template <typename RS> static int launch_guard_p(const GuardArgs<RS>& a, cudaStream_t st) {
  switch (padded_size(a.N)) {
    case 8: return launch_guard_t<RS, 8, 8>(a, st);
    case 16: return launch_guard_t<RS, 16, 4>(a, st);
    case 24: return launch_guard_t<RS, 24, 2>(a, st);
    case 32: return launch_guard_t<RS, 32, 1>(a, st);
    case 48: return launch_guard_t<RS, 48, 1>(a, st);
    default:
      set_last_error("basis size N_b=%d exceeds the supported maximum 48", a.N);
      return QCL_UNSUPPORTED;
  }
}

// The budgets use the unit roundoff of the storage precision (complex64
// fields carry FP32 rounding in every entry), or `roundoff` when that is
// larger: a state promoted from complex64 to complex128 still carries the
// FP32 rounding of the iterations that made it, and its near-zero
// eigenvalues sit at that level.
int launch_anderson_guard(int precision, int NE, int Nk, int N, void* const* fields, int nfam, AndersonMeta* m,
                          int pass, double roundoff, cudaStream_t st) {
  if (nfam < 1 || nfam > kGuardMaxFamilies) {
    set_last_error("anderson guard: %d families out of range", nfam);
    return QCL_ARG;
  }
  const double store_eps = precision == QCL_C128 ? 2.220446049250313e-16 : 1.1920928955078125e-07;
  const double eps = roundoff > store_eps ? roundoff : store_eps;
  if (precision == QCL_C128) {
    GuardArgs<double> a{NE, Nk, N, nfam, pass, eps, {}, m};
    for (int i = 0; i < 3 * nfam; ++i) a.f[i] = (const Cx<double>*)fields[i];
    return launch_guard_p<double>(a, st);
  }
  GuardArgs<float> a{NE, Nk, N, nfam, pass, eps, {}, m};
  for (int i = 0; i < 3 * nfam; ++i) a.f[i] = (const Cx<float>*)fields[i];
  return launch_guard_p<float>(a, st);
}


size_t residual_work_doubles(int NE, int Nk) { return kResidualBlockDoubles * (size_t)NE * Nk + 7 * RES_CTAS; }

// ---------------------------------------------------------------------------
// Allocation-free variant.  Some callers cannot call cudaMalloc: a Julia
// session whose device memory is owned by its own pool allocator, a host
// application that reserves a fixed device budget up front, or a solver loop
// that must not pay the device synchronisation an allocation can imply.  For
// them the residual suite's scratch (9 doubles per (E,k) block plus 7 per
// reduction CTA) lives in this file-scope device array instead.  Every GPU
// that loads the library holds it (about 18.9 MB) until the process exits.
// ---------------------------------------------------------------------------
constexpr long long kNoAllocMaxBlocks = 1ll << 18;  // N_E * N_k <= 262144
// the layout of residual_work_doubles(N_E, N_k) at N_E * N_k = kNoAllocMaxBlocks
constexpr long long kNoAllocScratchDoubles = kResidualBlockDoubles * kNoAllocMaxBlocks + 7ll * RES_CTAS;
static __device__ __align__(256) double g_residual_scratch[kNoAllocScratchDoubles];

static std::mutex g_noalloc_mutex;
static double* g_noalloc_ptr[64] = {nullptr};

// Device address of the scratch array on the current device, resolved once
// per device (host code cannot use the symbol itself as an address).  The
// address stays valid for the life of the device context: after a
// cudaDeviceReset (CUDA.jl's device_reset!) every device pointer held by the
// library is stale, this one included, and the entry point must not be used.
static int noalloc_scratch(double** out) {
  int dev = 0;
  QCL_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_last_error("device ordinal %d out of range", dev);
    return QCL_ARG;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_residual_scratch);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(g_residual_scratch)");
    g_noalloc_ptr[dev] = (double*)p;
  }
  *out = g_noalloc_ptr[dev];
  return QCL_OK;
}

// Per-block pass of the residual suite (part: RES_PART_ALL, or the two halves
// RES_PART_MAIN and RES_PART_RK, which write disjoint per-block slots and may
// run concurrently).
int launch_residual_blocks(int precision, int part, int NE, int Nk, int N, const double* eps, const void* h,
                           const void* GR, const void* GL, const void* GG, const void* SR, const void* SL,
                           const void* SG, const void* SLc, double* work, cudaStream_t st) {
  if (part != RES_PART_ALL && part != RES_PART_MAIN && part != RES_PART_RK) {
    set_last_error("residual suite: unknown part %d", part);
    return QCL_ARG;
  }
  if (precision == QCL_C128) {
    ResidualArgs<double> a{NE, Nk, N, eps, (const Cx<double>*)h, (const Cx<double>*)GR, (const Cx<double>*)GL,
                           (const Cx<double>*)GG, (const Cx<double>*)SR, (const Cx<double>*)SL,
                           (const Cx<double>*)SG, (const Cx<double>*)SLc, work, part};
    return launch_residual_p<double>(a, st);
  }
  ResidualArgs<float> a{NE, Nk, N, eps, (const Cx<double>*)h, (const Cx<float>*)GR, (const Cx<float>*)GL,
                        (const Cx<float>*)GG, (const Cx<float>*)SR, (const Cx<float>*)SL, (const Cx<float>*)SG,
                        (const Cx<float>*)SLc, work, part};
  return launch_residual_p<float>(a, st);
}

int launch_residual_suite(int precision, int NE, int Nk, int N, const double* eps, const void* h, const void* GR,
                          const void* GL, const void* GG, const void* SR, const void* SL, const void* SG,
                          const void* SLc, double* work, double* out5, cudaStream_t st) {
  int s = launch_residual_blocks(precision, RES_PART_ALL, NE, Nk, N, eps, h, GR, GL, GG, SR, SL, SG, SLc, work, st);
  if (s) return s;
  return launch_residual_reduce(NE, Nk, work, out5, st);
}

// The witness of the residual suite whose per-block outputs are in `work`
// (the same work array and fields as the launch_residual_suite call before
// it).  out12: kind, e, m, then minimum_eigenvalue, block_norm, floor, ratio,
// absolute_defect, relative_defect, backward_error, hermiticity_defect,
// construction_scale.  Uses 3 * RES_CTAS doubles of `partial` scratch.
int launch_residual_witness(int precision, int NE, int Nk, int N, const void* GR, const void* GL, const void* GG,
                            const void* SL, const void* SG, const double* work, double* partial, double* out12,
                            cudaStream_t st) {
  witness_reduce_kernel<<<RES_CTAS, 256, 0, st>>>((long long)NE * Nk, NE, Nk, work, partial);
  QCL_LAUNCH_CHECK("witness_reduce_kernel");
  if (precision == QCL_C128) {
    WitnessArgs<double> a{NE, Nk, N, RES_CTAS, (const Cx<double>*)GR, (const Cx<double>*)GL, (const Cx<double>*)GG,
                          (const Cx<double>*)SL, (const Cx<double>*)SG, partial, out12};
    return launch_witness_detail_p<double>(a, st);
  }
  WitnessArgs<float> a{NE, Nk, N, RES_CTAS, (const Cx<float>*)GR, (const Cx<float>*)GL, (const Cx<float>*)GG,
                       (const Cx<float>*)SL, (const Cx<float>*)SG, partial, out12};
  return launch_witness_detail_p<float>(a, st);
}

size_t residual_witness_partial_doubles() { return 3 * RES_CTAS; }

}  // namespace qcl

using namespace qcl;

// The scratch is fully rewritten by every call before it is read (each live
// block writes its 7 values, the reduction writes all its partials), so
// nothing needs clearing between calls.  Calls share the array: two calls that
// overlap on the GPU (different streams, or concurrent host threads) race on
// it.  The first call on a device resolves the array's address on that
// device; make that first call before any stream capture.
extern "C" int qcl_dev_residual_suite_noalloc(void* stream, int precision, int NE, int Nk, int Nb, const double* eps,
                                              const void* h, const void* GR, const void* GL, const void* GG,
                                              const void* SR, const void* SL, const void* SG, const void* SLc,
                                              double* out) {
  if (precision != QCL_C128 && precision != QCL_C64 && precision != QCL_MIXED) {
    set_last_error("unknown precision %d", precision);
    return QCL_ARG;
  }
  if (NE <= 0 || Nk <= 0 || Nb <= 0) {
    set_last_error("residual_suite_noalloc: non-positive dimension (%d,%d,%d)", NE, Nk, Nb);
    return QCL_DIM;
  }
  if ((long long)NE * Nk > kNoAllocMaxBlocks) {
    set_last_error("residual_suite_noalloc: N_E*N_k = %lld exceeds the fixed scratch capacity of %lld blocks",
                   (long long)NE * Nk, kNoAllocMaxBlocks);
    return QCL_UNSUPPORTED;
  }
  if (!eps || !h || !GR || !GL || !GG || !SR || !SL || !SG || !SLc || !out) {
    set_last_error("residual_suite_noalloc: all arrays are required");
    return QCL_ARG;
  }
  if ((long long)residual_work_doubles(NE, Nk) > kNoAllocScratchDoubles) {  // holds by the block limit above
    set_last_error("residual_suite_noalloc: scratch layout exceeds the fixed array");
    return QCL_UNSUPPORTED;
  }
  double* scratch = nullptr;
  int s = noalloc_scratch(&scratch);
  if (s) return s;
  const int sp = precision == QCL_MIXED ? QCL_C64 : precision;
  return launch_residual_suite(sp, NE, Nk, Nb, eps, h, GR, GL, GG, SR, SL, SG, SLc, scratch, out,
                               (cudaStream_t)stream);
}
