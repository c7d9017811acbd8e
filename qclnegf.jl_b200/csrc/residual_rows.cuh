// Residual suite kernels for N_b <= 32.
#pragma once
#include "residual.cuh"

namespace qcl {

// ---------------------------------------------------------------------------
// The suite for N_b <= 32.  Its seven positivity tests were most of the time
// of residual_kernel (which remains for N_b > 32): an LDL^T whose trailing block lives in
// shared memory, one matrix after another, half the lanes idle.  Here each
// LDL^T keeps one row per lane in registers, so a warp takes 32 / NP matrices
// at once (four at N_b <= 8, two at N_b <= 16; the two warps of an N_b <= 32
// team one each), reads their entries straight from the tiles of the fields
// they are made of, and exchanges one column per step.  Products whose result
// only enters a norm stay in registers, and G Gamma G^H of r_A is the
// difference of the two raw Keldysh products, which are formed anyway.
// Tests that fail are settled afterwards, with every tile free, by the
// tridiagonal reduction (psd_of, team_lmax).
// Bound by FP64 issue at 12 warps per SM.  mixed, 32 768 blocks: N_b = 16 2.16 -> 1.21
// ms, N_b = 32 20.0 -> 8.6 ms; complex128: 2.18 -> 1.31, 20.1 -> 11.5 ms.
// ---------------------------------------------------------------------------
enum { HK_A = 0, HK_GL = 1, HK_GG = 2, HK_GAM = 3, HK_RAWL = 4, HK_RAWG = 5, HK_CAUS = 6, HK_COUNT = 7 };

template <int NP> struct RowScratch {
  Cx<double> col[2][Tile<NP>::TT];  // column being eliminated, per matrix of a round
  unsigned fail[Tile<NP>::TT / 32], bad[Tile<NP>::TT / 32];
};

// Entry (i, j) of the Hermitian matrix of a test, from the tiles: G = G^R,
// X = Sigma^R (HK_CAUS), Sigma< (HK_GAM) or the raw lesser product (HK_RAWL),
// W = G< (HK_GL), Sigma> (HK_GAM) or the raw greater product, H = G> (HK_GG).
template <int NP>
__device__ __forceinline__ Cx<double> herm_entry(int kind, const Cx<double>* G, const Cx<double>* X, const Cx<double>* W,
                                                 const Cx<double>* H, int i, int j, bool& finite) {
  const int ij = sw<NP>(i, j), ji = sw<NP>(j, i);
  if (kind == HK_GAM) {  // i (S> - S<)
    const Cx<double> g = W[ij], l = X[ij], gt = W[ji], lt = X[ji];
    const double x = g.x - l.x, y = g.y - l.y, xt = gt.x - lt.x, yt = gt.y - lt.y;
    finite = finite && isfinite(x) && isfinite(y) && isfinite(xt) && isfinite(yt);
    return cx<double>(0.5 * (-y - yt), 0.5 * (x - xt));
  }
  const Cx<double>* T = kind == HK_A ? G : kind == HK_GL || kind == HK_RAWG ? W : kind == HK_GG ? H : X;
  const Cx<double> a = T[ij], b = T[ji];
  finite = finite && isfinite(a.x) && isfinite(a.y) && isfinite(b.x) && isfinite(b.y);
  if (kind == HK_A) return cx<double>(-(a.y + b.y), a.x - b.x);                        // i (G - G^H)
  if (kind == HK_CAUS) return cx<double>(-0.5 * (a.y + b.y), 0.5 * (a.x - b.x));       // -Im_H Sigma^R
  if (kind == HK_GL || kind == HK_RAWL) return cx<double>(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));  // -i X
  return cx<double>(-0.5 * (a.y + b.y), 0.5 * (a.x - b.x));                            // i X
}

// LDL^T tests of the matrices `kinds` (4 bits each, `count` of them): bit k of
// fail / bad is set when matrix kind k has no certificate / is not finite.
// Every thread of the team returns the same masks.
template <int NP, int TT>
__device__ void posdef_rounds(unsigned kinds, int count, const Cx<double>* G, const Cx<double>* X, const Cx<double>* W,
                              const Cx<double>* H, int N, int tt, RowScratch<NP>& R, int team, unsigned& fail,
                              unsigned& bad) {
  constexpr int PER = TT / NP;  // matrices per round
  constexpr double eps = 2.220446049250313e-16;
  unsigned f = 0, b = 0;
#pragma unroll 1
  for (int base = 0; base < count; base += PER) {
    const int g = tt / NP, r = tt - g * NP, q = base + g;
    const bool mine = g < PER && q < count;
    const int kind = mine ? (int)((kinds >> (4 * q)) & 15u) : HK_A;
    Cx<double> row[NP];
    bool finite = true;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      row[j] = cx<double>(j == r ? 1.0 : 0.0, 0.0);
      if (mine && j <= r && r < N) row[j] = herm_entry<NP>(kind, G, X, W, H, r, j, finite);
    }
    double d = 0.0;  // largest diagonal entry of the matrix
#pragma unroll
    for (int j = 0; j < NP; ++j)
      if (j == r && r < N) d = fabs(row[j].x);
    Cx<double>* col = R.col[0] + g * NP;
    // (lanes past the last matrix use the tail of the buffers)
    if (PER * NP == TT || g < PER) col[r] = cx<double>(d, finite ? 0.0 : 1.0);
    __syncwarp();
    double nonfin = 0.0;
    d = 0.0;
    if (g < PER)
      for (int j = 0; j < N; ++j) {
        const Cx<double> c = col[j];
        d = fmax(d, c.x);
        nonfin += c.y;
      }
    const double shift = kind == HK_CAUS ? 0.0 : 64.0 * N * eps * fmax(d, 1.0);
    bool ok = true;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      if (k >= N) break;
      Cx<double>* c = R.col[k & 1] + g * NP;
      if (g < PER) c[r] = row[k];
      __syncwarp();
      if (g < PER) {
        const double dk = c[k].x + shift;
        ok = ok && dk > 0;
        const double inv = 1.0 / dk;
        const Cx<double> l = cx<double>(row[k].x * inv, row[k].y * inv);
#pragma unroll
        for (int j = k + 1; j < NP; ++j) {
          const Cx<double> a = c[j];  // row[j] -= l conj(a)
          row[j].x = fma(-l.x, a.x, row[j].x);
          row[j].x = fma(-l.y, a.y, row[j].x);
          row[j].y = fma(l.x, a.y, row[j].y);
          row[j].y = fma(-l.y, a.x, row[j].y);
        }
      }
    }
    __syncwarp();
    if (mine && r == 0) {
      if (nonfin != 0.0) b |= 1u << kind;
      else if (!ok) f |= 1u << kind;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    f |= __shfl_xor_sync(0xffffffffu, f, o);
    b |= __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (TT > 32) {
    team_sync<TT>(team);
    if ((tt & 31) == 0) {
      R.fail[tt >> 5] = f;
      R.bad[tt >> 5] = b;
    }
    team_sync<TT>(team);
    f = b = 0;
#pragma unroll
    for (int w = 0; w < TT / 32; ++w) {
      f |= R.fail[w];
      b |= R.bad[w];
    }
  }
  fail |= f;
  bad |= b;
}

// Loads the tiles of `count` fields with all their accesses in flight.
template <typename RS, int NP, int BPC, size_t STRIDE, int COUNT>
__device__ __forceinline__ void load_tiles(const Cx<RS>* const (&src)[COUNT], Cx<double>* const (&dst)[COUNT], int e0,
                                           int m, int NE, int Nk, int N) {
  constexpr int IT = NP * NP / Tile<NP>::TT;
  static_assert(IT * Tile<NP>::TT == NP * NP, "tile size");
  const size_t base = (size_t)e0 + (size_t)NE * m, cstride = (size_t)NE * Nk;
  const int eloc = threadIdx.x % BPC;
  const bool ein = e0 + eloc < NE;
  constexpr int G = IT % 4 == 0 ? 4 : IT % 3 == 0 ? 3 : IT;  // elements per field in flight
#pragma unroll 1
  for (int q0 = 0; q0 < IT; q0 += G) {
    Cx<RS> v[COUNT][G];
#pragma unroll
    for (int f = 0; f < COUNT; ++f)
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int el = (threadIdx.x + (q0 + q) * BPC * Tile<NP>::TT) / BPC, a = el % NP, b = el / NP;
        v[f][q] = cx<RS>(0, 0);
        if (ein && a < N && b < N) v[f][q] = src[f][base + eloc + cstride * ((size_t)a + (size_t)N * b)];
      }
#pragma unroll
    for (int f = 0; f < COUNT; ++f)
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int el = (threadIdx.x + (q0 + q) * BPC * Tile<NP>::TT) / BPC;
        dst[f][eloc * STRIDE + sw<NP>(el % NP, el / NP)] = cvt<double>(v[f][q]);
      }
  }
}

// Visits the accumulators of a team product: f(row, column, value), within N.
template <int NP, int TT, typename F>
__device__ __forceinline__ void acc_for(const DmmaTile<NP, TT>& acc, int N, int tt, F&& f) {
  constexpr int NT = DmmaTile<NP, TT>::NT, NW = DmmaTile<NP, TT>::NW, RPW = DmmaTile<NP, TT>::RPW;
  const int warp = tt >> 5, lane = tt & 31, lr = lane >> 2, lc = lane & 3;
#pragma unroll
  for (int r = 0; r < RPW; ++r)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int a = (warp + r * NW) * 8 + lr, b = j * 8 + 2 * lc + i;
        if (a < N && b < N) f(a, b, cx<double>(acc.re[r][j][i], acc.im[r][j][i]));
      }
}

// sum |K - G S G^H|^2 and sum |K|^2 with S in tile T (overwritten by G S).
template <int NP, int TT>
__device__ void keldysh_defect(const Cx<double>* G, Cx<double>* T, const Cx<double>* K, int N, int tt, double* scratch,
                               int team, double& num, double& den) {
  DmmaTile<NP, TT> acc;
  team_matmul_dmma<NP, TT>(G, T, acc, N, tt, false);
  team_sync<TT>(team);
  team_store_dmma<NP, TT>(T, acc, tt);
  team_sync<TT>(team);
  team_matmul_dmma<NP, TT>(T, G, acc, N, tt, true);
  num = den = 0;
  acc_for<NP, TT>(acc, N, tt, [&](int i, int j, Cx<double> q) {
    const Cx<double> a = K[sw<NP>(i, j)];
    num += (a.x - q.x) * (a.x - q.x) + (a.y - q.y) * (a.y - q.y);
    den += a.x * a.x + a.y * a.y;
  });
  team_sum2<TT>(num, den, tt, scratch, team);
}

// r_K alone (RES_PART_RK).
template <typename RS, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT) residual_rk_kernel(ResidualArgs<RS> p) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = tile_stride<double, NP, BPC>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bG = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* bX = bG + BPC * MSZ;
  Cx<double>* bW = bX + BPC * MSZ;
  double* red = reinterpret_cast<double*>(bW + BPC * MSZ);
  const int N = p.N, NE = p.NE, Nk = p.Nk, m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT, e = e0 + team;
  load_tiles<RS, NP, BPC, MSZ, 3>({p.GR, p.GL, p.SLc}, {bG, bX, bW}, e0, m, NE, Nk, N);
  __syncthreads();
  double kNum, kDen;
  keldysh_defect<NP, TT>(bG + team * MSZ, bW + team * MSZ, bX + team * MSZ, N, tt, red + 4 * team, team, kNum, kDen);
  if (tt == 0 && e < NE) {
    double* o = p.block_out + kResidualBlockDoubles * ((size_t)e + (size_t)NE * m);
    o[3] = isfinite(kNum) ? kNum : INFINITY;
    o[4] = isfinite(kDen) ? kDen : INFINITY;
  }
}

// Up to N_b = 16 registers bound the CTAs per SM, so a fourth tile is free and
// saves a load and a round of tests (N_b = 12: 0.95 against 1.05 ms); above,
// three tiles give the fourth CTA (N_b = 32, mixed: 17.4 against 8.6 ms).
template <int NP> constexpr bool rows_four_tiles() { return NP <= 16; }
// Register budget: the CTAs per SM that the tiles' shared memory allows (168
// registers at N_b <= 16; 128 there spill: 1.24 -> 1.47 ms).
template <int NP> constexpr int rows_min_ctas() { return NP == 8 ? 2 : NP == 16 ? 6 : NP == 32 ? 4 : 3; }

template <typename RS, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT, (rows_min_ctas<NP>())) residual_rows_kernel(ResidualArgs<RS> p) {
  constexpr bool FOUR = rows_four_tiles<NP>();
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = (size_t)NP * NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* bG = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* bX = bG + BPC * MSZ;
  Cx<double>* bW = bX + BPC * MSZ;
  Cx<double>* bH = FOUR ? bW + BPC * MSZ : bX;
  RowScratch<NP>* rows = reinterpret_cast<RowScratch<NP>*>((FOUR ? bH : bW) + BPC * MSZ);
  ResScratch<NP>* scr = reinterpret_cast<ResScratch<NP>*>(rows + BPC);
  const int N = p.N, NE = p.NE, Nk = p.Nk, m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT, e = e0 + team;
  const bool live = e < NE;
  Cx<double>* G = bG + team * MSZ;
  Cx<double>* X = bX + team * MSZ;
  Cx<double>* W = bW + team * MSZ;
  const Cx<double>* H = bH + team * MSZ;
  RowScratch<NP>& R = rows[team];
  ResScratch<NP>& S = scr[team];
  unsigned fail = 0, bad = 0;
  auto kinds = [](int a, int b = 0, int c = 0, int d = 0) { return (unsigned)(a | b << 4 | c << 8 | d << 12); };

  // ---- causality, A ---------------------------------------------------------
  if constexpr (FOUR) load_tiles<RS, NP, BPC, MSZ, 4>({p.GR, p.SR, p.GL, p.GG}, {bG, bX, bW, bH}, e0, m, NE, Nk, N);
  else load_tiles<RS, NP, BPC, MSZ, 3>({p.GR, p.SR, p.GL}, {bG, bX, bW}, e0, m, NE, Nk, N);
  __syncthreads();
  posdef_rounds<NP, TT>(kinds(HK_CAUS, HK_A, HK_GL, HK_GG), FOUR ? 4 : 2, G, X, W, H, N, tt, R, team, fail, bad);
  team_sync<TT>(team);

  DmmaTile<NP, TT> acc;
  // ---- r_D: D over Sigma^R, ||D G - I|| from the accumulators ---------------
  const double eps_e = live ? p.eps[e] : 0.0;
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
  team_matmul_dmma<NP, TT>(X, G, acc, N, tt, false);
  double nR = 0;
  acc_for<NP, TT>(acc, N, tt, [&](int i, int j, Cx<double> v) {
    if (i == j) v.x -= 1;
    nR += v.x * v.x + v.y * v.y;
  });
  nR = team_sum<TT>(nR, tt, S.red, team);
  double rD = sqrt(nR) / (sqrt(nD) * sqrt(nG) + sqrt((double)N));
  if (!isfinite(rD)) rD = INFINITY;

  // ---- r_K ------------------------------------------------------------------
  const bool with_rk = p.part == RES_PART_ALL;  // launch-uniform
  double kNum = 0, kDen = 0;
  if (with_rk) {
    __syncthreads();
    load_tiles<RS, NP, BPC, MSZ, 1>({p.SLc}, {bX}, e0, m, NE, Nk, N);
    __syncthreads();
    keldysh_defect<NP, TT>(G, X, W, N, tt, S.red, team, kNum, kDen);
  }

  // ---- G<, G>, Gamma, then the raw products ---------------------------------
  __syncthreads();
  if constexpr (!FOUR) {
    load_tiles<RS, NP, BPC, MSZ, 1>({p.GG}, {bX}, e0, m, NE, Nk, N);
    __syncthreads();
    posdef_rounds<NP, TT>(kinds(HK_GL, HK_GG), 2, G, X, W, H, N, tt, R, team, fail, bad);
    __syncthreads();
  }
  load_tiles<RS, NP, BPC, MSZ, 2>({p.SL, p.SG}, {bX, bW}, e0, m, NE, Nk, N);
  __syncthreads();
  posdef_rounds<NP, TT>(kinds(HK_GAM), 1, G, X, W, H, N, tt, R, team, fail, bad);
  team_sync<TT>(team);
  auto sandwich = [&](Cx<double>* T) {  // T <- G T G^H
    team_matmul_dmma<NP, TT>(G, T, acc, N, tt, false);
    team_sync<TT>(team);
    team_store_dmma<NP, TT>(T, acc, tt);
    team_sync<TT>(team);
    team_matmul_dmma<NP, TT>(T, G, acc, N, tt, true);
    team_sync<TT>(team);
    team_store_dmma<NP, TT>(T, acc, tt);
    team_sync<TT>(team);
  };
  sandwich(X);
  sandwich(W);
  posdef_rounds<NP, TT>(kinds(HK_RAWL, HK_RAWG), 2, G, X, W, H, N, tt, R, team, fail, bad);
  // ---- r_A: A - G Gamma G^H = A - i (raw> - raw<) ---------------------------
  double aNum = 0, aDen = 0;
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> g = G[sw<NP>(i, j)], gt = G[sw<NP>(j, i)], rl = X[sw<NP>(i, j)], rg = W[sw<NP>(i, j)];
    const double ax = -(g.y + gt.y), ay = g.x - gt.x;
    const double dx = ax + (rg.y - rl.y), dy = ay - (rg.x - rl.x);
    aNum += dx * dx + dy * dy;
    aDen += ax * ax + ay * ay;
  });
  team_sum2<TT>(aNum, aDen, tt, S.red, team);

  // ---- tests without a certificate ------------------------------------------
  double psd = 0, wr = -1.0, wk = -1.0;  // as in residual_kernel
  double caus = bad >> HK_CAUS & 1u ? INFINITY : 0.0;
  const Cx<double> one = cx<double>(1, 0), mi = cx<double>(0, -1), pi = cx<double>(0, 1);
#pragma unroll 1
  for (int kind = 0; kind < 6; ++kind) {
    double r = bad >> kind & 1u ? INFINITY : 0.0;
    // a CTA's blocks reload together: the loads are CTA-wide
    const bool need = (fail >> kind & 1u) && live;
    if (__syncthreads_or(need)) {
      const Cx<RS>* src = kind == HK_A ? p.GR : kind == HK_GL ? p.GL : kind == HK_GG ? p.GG : kind == HK_RAWG ? p.SG : p.SL;
      load_tiles<RS, NP, BPC, MSZ, 1>({src}, {bX}, e0, m, NE, Nk, N);
      if (kind == HK_GAM) load_tiles<RS, NP, BPC, MSZ, 1>({p.SG}, {bW}, e0, m, NE, Nk, N);
      __syncthreads();
      if (need) {
        if (kind == HK_RAWL || kind == HK_RAWG) sandwich(X);
        if (kind == HK_A || kind == HK_GAM) {
          tile_for<NP, TT>(N, tt, [&](int i, int j) {
            const Cx<double> g = kind == HK_A ? G[sw<NP>(i, j)] : W[sw<NP>(i, j)];
            const Cx<double> l = kind == HK_A ? conj(G[sw<NP>(j, i)]) : X[sw<NP>(i, j)];
            X[sw<NP>(i, j)] = pi * cx<double>(g.x - l.x, g.y - l.y);
          });
          team_sync<TT>(team);
        }
        r = psd_of<NP, TT>(X, kind == HK_GL || kind == HK_RAWL ? mi : kind == HK_GG || kind == HK_RAWG ? pi : one, W, N,
                           tt, S, team);
        team_sync<TT>(team);
      }
    }
    psd = fmax(psd, r);
    if (kind >= 4 && !isfinite(r)) continue;
    if (r > wr) {  // kinds in ascending order: the lowest kind keeps a tie
      wr = r;
      wk = kind;
    }
  }
  const bool need = (fail >> HK_CAUS & 1u) && live;
  if (__syncthreads_or(need)) {
    load_tiles<RS, NP, BPC, MSZ, 1>({p.SR}, {bX}, e0, m, NE, Nk, N);
    __syncthreads();
    if (need) {
      tile_for<NP, TT>(N, tt, [&](int i, int j) {
        const Cx<double> a = X[sw<NP>(i, j)], b = X[sw<NP>(j, i)];
        W[sw<NP>(i, j)] = cx<double>(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));  // (a - conj(b)) / (2i)
      });
      team_sync<TT>(team);
      const double num = fmax(0.0, team_lmax<NP, TT>(W, N, tt, S, team, true));
      team_sync<TT>(team);
      if (num > 0 && isfinite(num)) {  // ||Sigma^R||_2^2 = lmax(Sigma^R Sigma^R^H)
        team_matmul<double, double, NP>(X, X, W, N, tt, true);
        team_sync<TT>(team);
        const double lmax = team_lmax<NP, TT>(W, N, tt, S, team, false);
        caus = num / (sqrt(fmax(lmax, 0.0)) + 1e-14);
      } else if (!isfinite(num)) {
        caus = INFINITY;
      }
    }
  }

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

// r_K alone has no tests and is bound by its loads, where longer runs of
// energies help: N_b = 32, 1024 x 32 blocks, mixed, 2 per CTA instead of 1: 1.52
// -> 0.98 ms; N_b = 12 and 16, 4 instead of 2: 6400 blocks, c128, 37 -> 30 us,
// 3064 blocks, mixed, 30 -> 24 us, and whole iterations at 3064 ... 32768 blocks
// take the same or less at every count (N_b = 16, c128: 484.9 -> 482.4 us at
// 3064, 1056 -> 1043 at 8192, 1987 -> 1960 at 16384, 3786 -> 3732 at 32768).
template <typename RS, int NP, int BPC> static int launch_residual_rk_t(const ResidualArgs<RS>& a, cudaStream_t st) {
  constexpr size_t smem = BPC * (3 * tile_stride<double, NP, BPC>() * sizeof(Cx<double>) + 4 * sizeof(double));
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(residual_rk_kernel<RS, NP, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  residual_rk_kernel<RS, NP, BPC><<<dim3((a.NE + BPC - 1) / BPC, a.Nk), BPC * Tile<NP>::TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("residual_rk_kernel");
  return QCL_OK;
}

template <typename RS, int NP, int BPC> static int launch_residual_rows_t(const ResidualArgs<RS>& a, cudaStream_t st) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t tile = (size_t)BPC * NP * NP * sizeof(Cx<double>);
  constexpr size_t smem = (rows_four_tiles<NP>() ? 4 : 3) * tile + BPC * (sizeof(RowScratch<NP>) + sizeof(ResScratch<NP>));
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(residual_rows_kernel<RS, NP, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  if (a.part == RES_PART_RK) {
    if (NP == 32) return launch_residual_rk_t<RS, NP, 2>(a, st);
    return launch_residual_rk_t<RS, NP, NP == 16 ? 4 : BPC>(a, st);
  }
  const dim3 grid((a.NE + BPC - 1) / BPC, a.Nk);
  residual_rows_kernel<RS, NP, BPC><<<grid, BPC * TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("residual_rows_kernel");
  return QCL_OK;
}

}  // namespace qcl
