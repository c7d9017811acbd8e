// Device routines of the residual suite that its kernels and those of the
// other spectral tests share: Hermitian parts, LDL^T tests, tridiagonal
// reduction, extreme eigenvalues, full spectra.
#pragma once
#include "blockmat.cuh"

namespace qcl {

// Per-block outputs: r_D, r_A num/den, r_K num/den, r_PSD, r_caus, and the
// block's positivity-witness ratio and matrix kind.
constexpr int kResidualBlockDoubles = 9;
constexpr int RES_CTAS = 148;  // of the reduction over blocks

template <typename RS> struct ResidualArgs {
  int NE, Nk, N;
  const double* eps;
  const Cx<double>* h;
  const Cx<RS>* GR;
  const Cx<RS>* GL;
  const Cx<RS>* GG;
  const Cx<RS>* SR;   // totals
  const Cx<RS>* SL;
  const Cx<RS>* SG;
  const Cx<RS>* SLc;  // candidate total lesser
  double* block_out;  // kResidualBlockDoubles per block
  int part;           // RES_PART_ALL, RES_PART_MAIN (all but r_K) or RES_PART_RK (r_K only)
};

struct JacobiRot {
  double c, s, pr, pi;  // rotation cosine/sine and the phase e^{i phi}
  int p, q;
};

template <int NP> struct ResScratch {
  JacobiRot rot[NP / 2];
  double red[8];
  double vals[NP];
  double d[NP], e2[NP];  // tridiagonal form
  Cx<double> u[NP], w[NP];
};

// Visits the (i, j), i, j < N, of an NP x NP tile: team thread tt takes the
// padded indices tt, tt + TT, ... (compile-time trip count and index split,
// no runtime division).
template <int NP, int TT, typename F> __device__ __forceinline__ void tile_for(int N, int tt, F&& f) {
#pragma unroll 1
  for (int q = 0; q < (NP * NP + TT - 1) / TT; ++q) {
    const int idx = tt + q * TT;
    if (idx < NP * NP) {
      const int i = idx % NP, j = idx / NP;
      if (i < N && j < N) f(i, j);
    }
  }
}

// Team sum of two doubles (fixed order).
template <int TT>
__device__ __forceinline__ void team_sum2(double& a, double& b, int tt, double* scratch, int team) {
  a = team_sum<TT>(a, tt, scratch, team);
  b = team_sum<TT>(b, tt, scratch + 2, team);
}

// Eigenvalues of the Hermitian NxN matrix H (swizzled NP x NP shared tile);
// H is destroyed, S.vals[0..N-1] receives the eigenvalues (unsorted).
// Round-robin parallel Jacobi: in each of the n2-1 rounds of a sweep the
// rotations of n2/2 disjoint index pairs are computed from the same matrix
// and applied together (all column updates, then all row updates).  The
// rotated pair is set to exactly zero and its diagonal to exactly real, so
// rounding cannot leave a non-Hermitian remainder; a pair whose coupling is
// negligible against its diagonal (1e-18 relative) is skipped, and a sweep
// that rotates nothing ends the iteration.
template <int NP, int TT>
__device__ void team_eigvals(Cx<double>* H, int N, int tt, ResScratch<NP>& S, int team) {
  const int n2 = N + (N & 1);
  for (int sweep = 0; sweep < 40; ++sweep) {
    double rotated = 0;
    for (int r = 0; r < n2 - 1; ++r) {
      if (tt < n2 / 2) {
        const int i = tt;
        const int a = (r + i) % (n2 - 1);
        const int b = (i == 0) ? n2 - 1 : (r - i + n2 - 1) % (n2 - 1);
        JacobiRot rt;
        rt.p = a < b ? a : b;
        rt.q = a < b ? b : a;
        rt.c = 1;
        rt.s = 0;
        rt.pr = 1;
        rt.pi = 0;
        if (rt.q < N) {
          const Cx<double> apq = H[sw<NP>(rt.p, rt.q)];
          const double mag = hypot(apq.x, apq.y);
          const double app = H[sw<NP>(rt.p, rt.p)].x, aqq = H[sw<NP>(rt.q, rt.q)].x;
          if (mag > 1e-18 * (fabs(app) + fabs(aqq)) && isfinite(mag)) {
            const double theta = (aqq - app) / (2 * mag);
            double t;
            if (fabs(theta) > 1e150) t = 0.5 / theta;
            else t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            rt.c = 1.0 / sqrt(t * t + 1.0);
            rt.s = t * rt.c;
            rt.pr = apq.x / mag;
            rt.pi = apq.y / mag;
            rotated = 1;
          }
        } else {
          rt.q = rt.p;  // phantom partner: identity
        }
        S.rot[i] = rt;
      }
      team_sync<TT>(team);
      // columns: H <- H J
      for (int idx = tt; idx < N * (n2 / 2); idx += TT) {
        const int k = idx % N;
        const JacobiRot rt = S.rot[idx / N];
        if (rt.p == rt.q || rt.s == 0) continue;
        const Cx<double> hp = H[sw<NP>(k, rt.p)], hq = H[sw<NP>(k, rt.q)];
        const Cx<double> eq = cx<double>(rt.pr, -rt.pi) * hq;  // e^{-i phi} H[k][q]
        H[sw<NP>(k, rt.p)] = cx<double>(rt.c * hp.x - rt.s * eq.x, rt.c * hp.y - rt.s * eq.y);
        H[sw<NP>(k, rt.q)] = cx<double>(rt.s * hp.x + rt.c * eq.x, rt.s * hp.y + rt.c * eq.y);
      }
      team_sync<TT>(team);
      // rows: H <- J^H H; the rotated pair becomes exactly diagonal
      for (int idx = tt; idx < N * (n2 / 2); idx += TT) {
        const int k = idx % N;
        const JacobiRot rt = S.rot[idx / N];
        if (rt.p == rt.q || rt.s == 0) continue;
        const Cx<double> xp = H[sw<NP>(rt.p, k)], xq = H[sw<NP>(rt.q, k)];
        const Cx<double> eq = cx<double>(rt.pr, rt.pi) * xq;  // e^{i phi} H[q][k]
        Cx<double> np_ = cx<double>(rt.c * xp.x - rt.s * eq.x, rt.c * xp.y - rt.s * eq.y);
        Cx<double> nq_ = cx<double>(rt.s * xp.x + rt.c * eq.x, rt.s * xp.y + rt.c * eq.y);
        if (k == rt.p) {
          np_.y = 0;             // H[p][p] real
          nq_ = cx<double>(0, 0);  // H[q][p] = 0
        } else if (k == rt.q) {
          np_ = cx<double>(0, 0);  // H[p][q] = 0
          nq_.y = 0;             // H[q][q] real
        }
        H[sw<NP>(rt.p, k)] = np_;
        H[sw<NP>(rt.q, k)] = nq_;
      }
      team_sync<TT>(team);
    }
    rotated = team_max<TT>(rotated, tt, S.red, team);
    if (rotated == 0) break;
  }
  for (int i = tt; i < N; i += TT) S.vals[i] = H[sw<NP>(i, i)].x;
  team_sync<TT>(team);
}

// Writes the Hermitian part of f*X into H; returns false if X has non-finite
// entries (team-uniform).
template <int NP, int TT>
__device__ bool hermitian_part(const Cx<double>* X, Cx<double> f, Cx<double>* H, int N, int tt, ResScratch<NP>& S,
                               int team) {
  double bad = 0;
  tile_for<NP, TT>(N, tt, [&](int i, int j) {
    const Cx<double> v = f * X[sw<NP>(i, j)], w = f * X[sw<NP>(j, i)];
    if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(w.x) || !isfinite(w.y)) bad = 1;
    H[sw<NP>(i, j)] = cx<double>(0.5 * (v.x + w.x), 0.5 * (v.y - w.y));
  });
  bad = team_max<TT>(bad, tt, S.red, team);
  team_sync<TT>(team);  // H complete for every thread of the team
  return bad == 0;
}

// ---- extreme eigenvalues through a tridiagonal form ---------------------------
// Householder reduction of the Hermitian N x N tile H (destroyed) to a real
// symmetric tridiagonal matrix with the same eigenvalues: S.d[0..N) its
// diagonal, S.e2[0..N-1) its squared off-diagonal.  Step k applies the
// Hermitian unitary reflector P = I - c u u^H that maps column k below the
// diagonal onto its first entry, as the rank-2 update of the trailing block
//   A <- P A P = A - u w^H - w u^H,  p = c A u,  w = p - (c/2)(u^H p) u
// (Golub & Van Loan, Matrix Computations, sec. 8.3.1).  One team thread per
// row of the trailing block; backward stable like LAPACK's zhetrd.
template <int NP, int TT>
__device__ void team_tridiagonalize(Cx<double>* H, int N, int tt, ResScratch<NP>& S, int team) {
  for (int k = 0; k + 2 < N; ++k) {
    const int m = N - k - 1;  // entries below the diagonal in column k
    const Cx<double> xi = tt < m ? H[sw<NP>(k + 1 + tt, k)] : cx<double>(0, 0);
    const double a2 = team_sum<TT>(xi.x * xi.x + xi.y * xi.y, tt, S.red, team);
    const Cx<double> x0 = H[sw<NP>(k + 1, k)];
    if (tt == 0) {
      S.d[k] = H[sw<NP>(k, k)].x;
      S.e2[k] = a2;
    }
    if (!(a2 > 0)) {  // team-uniform: column already reduced
      team_sync<TT>(team);
      continue;
    }
    const double alpha = sqrt(a2), ax0 = hypot(x0.x, x0.y);
    const Cx<double> ph = ax0 > 0 ? cx<double>(x0.x / ax0, x0.y / ax0) : cx<double>(1, 0);
    const double c = 1.0 / (alpha * (alpha + ax0));
    const Cx<double> ui = tt == 0 ? cx<double>(x0.x + alpha * ph.x, x0.y + alpha * ph.y) : xi;
    if (tt < m) S.u[tt] = ui;
    team_sync<TT>(team);
    Cx<double> pv = cx<double>(0, 0);
    if (tt < m) {
      for (int j = 0; j < m; ++j) cfma(pv, H[sw<NP>(k + 1 + tt, k + 1 + j)], S.u[j]);
      pv = c * pv;
    }
    const double kk = 0.5 * c * team_sum<TT>(tt < m ? ui.x * pv.x + ui.y * pv.y : 0.0, tt, S.red, team);
    if (tt < m) S.w[tt] = cx<double>(pv.x - kk * ui.x, pv.y - kk * ui.y);
    team_sync<TT>(team);
    for (int idx = tt; idx < m * m; idx += TT) {
      const int i = idx % m, j = idx / m;
      Cx<double>& a = H[sw<NP>(k + 1 + i, k + 1 + j)];
      const Cx<double> t = S.u[i] * conj(S.w[j]) + S.w[i] * conj(S.u[j]);
      a = cx<double>(a.x - t.x, a.y - t.y);
    }
    team_sync<TT>(team);
  }
  if (tt == 0) {
    if (N >= 2) {
      const Cx<double> t = H[sw<NP>(N - 1, N - 2)];
      S.d[N - 2] = H[sw<NP>(N - 2, N - 2)].x;
      S.e2[N - 2] = t.x * t.x + t.y * t.y;
    }
    S.d[N - 1] = H[sw<NP>(N - 1, N - 1)].x;
  }
  team_sync<TT>(team);
}

// Number of eigenvalues of the tridiagonal (d, e2) below sigma (Sturm
// sequence / LDL^T inertia, pivots clamped away from zero as in LAPACK dstebz).
__device__ __forceinline__ int sturm_count(const double* d, const double* e2, int N, double sigma, double pivmin) {
  double q = d[0] - sigma;
  if (fabs(q) < pivmin) q = -pivmin;
  int c = q < 0;
  for (int i = 1; i < N; ++i) {
    q = (d[i] - sigma) - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    c += q < 0;
  }
  return c;
}

__device__ __forceinline__ double tri_pivmin(const double* e2, int N) {
  double emax = 0;
  for (int i = 0; i + 1 < N; ++i) emax = fmax(emax, e2[i]);
  return 2.2250738585072014e-308 * fmax(1.0, emax);
}

// kth smallest eigenvalue (kth = 1..N) of the tridiagonal by multisection of
// the Gershgorin interval: each warp evaluates the same 32 shifts per round
// (every lane of the team ends with the same interval, no exchange needed),
// until the interval is a few ulps wide.
static __device__ double tri_eig(const double* d, const double* e2, int N, int kth) {
  constexpr double eps = 2.220446049250313e-16;
  double lo = INFINITY, hi = -INFINITY;
  for (int i = 0; i < N; ++i) {
    const double r = (i > 0 ? sqrt(e2[i - 1]) : 0.0) + (i + 1 < N ? sqrt(e2[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
  }
  const double pivmin = tri_pivmin(e2, N);
  const double tnorm = fmax(fabs(lo), fabs(hi));
  lo -= 2 * eps * tnorm * N + 2 * pivmin;
  hi += 2 * eps * tnorm * N + 2 * pivmin;
  const int lane = threadIdx.x & 31;
  for (int round = 0; round < 64; ++round) {
    if (hi - lo <= 2 * eps * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    const double width = hi - lo;
    const double sig = lo + width * (double)(lane + 1) / 33.0;
    const unsigned mask = __ballot_sync(0xffffffffu, sturm_count(d, e2, N, sig, pivmin) >= kth);
    const int f = mask ? __ffs(mask) - 1 : 32;  // first shift with kth eigenvalues below it
    const double nlo = f > 0 ? lo + width * (double)f / 33.0 : lo;
    const double nhi = f < 32 ? lo + width * (double)(f + 1) / 33.0 : hi;
    lo = nlo;
    hi = nhi;
  }
  return 0.5 * (lo + hi);
}

// True if H + shift I is numerically positive definite: LDL^T without pivoting
// (trailing lower triangle updated in place) meets only positive pivots.  H is
// destroyed.  A success certifies lmin(H) > -shift up to the factorization's
// backward error O(n eps ||H||) -- the same order as the error of the
// eigenvalues themselves.
template <int NP, int TT>
__device__ bool team_posdef(Cx<double>* H, int N, double shift, int tt, int team) {
  // TT / NP threads per row (rows past the tile's thread count idle): thread
  // (i, h) updates entries j = k + 1 + h, k + 1 + h + R, ... <= i of row i
  constexpr int R = TT / NP >= 1 ? TT / NP : 1;
  const int i = tt % NP, h = tt / NP;
  for (int k = 0; k < N; ++k) {
    const double dk = H[sw<NP>(k, k)].x + shift;
    if (!(dk > 0)) return false;  // team-uniform: every thread read the same pivot
    const double inv = 1.0 / dk;
    if (h < R && i > k && i < N) {
      const Cx<double> a = H[sw<NP>(i, k)];
      for (int j = k + 1 + h; j <= i; j += R) {
        const Cx<double> b = H[sw<NP>(j, k)];
        Cx<double>& hij = H[sw<NP>(i, j)];
        const Cx<double> t = a * conj(b);
        hij = cx<double>(hij.x - inv * t.x, hij.y - inv * t.y);
      }
    }
    team_sync<TT>(team);
  }
  return true;
}

// Positivity ratio of the Hermitian part of f X (written to H, destroyed):
//   max(0, -lmin - 64 n eps max(|l|max, 1)) / |l|max,
// INFINITY if f X has non-finite entries.  The diagonal bounds |l|max from
// below, so when H + 64 n eps max(max|H_ii|, 1) I is positive definite (one
// LDL^T, the common case) the ratio is 0; otherwise H is rebuilt, reduced to
// tridiagonal form and lmin, lmax are found by multisection.
template <int NP, int TT>
__device__ double psd_of(const Cx<double>* X, Cx<double> f, Cx<double>* H, int N, int tt, ResScratch<NP>& S,
                         int team) {
  constexpr double eps = 2.220446049250313e-16;
  if (!hermitian_part<NP, TT>(X, f, H, N, tt, S, team)) return INFINITY;
  double dmax = 0;
  for (int i = 0; i < N; ++i) dmax = fmax(dmax, fabs(H[sw<NP>(i, i)].x));
  team_sync<TT>(team);
  if (team_posdef<NP, TT>(H, N, 64.0 * N * eps * fmax(dmax, 1.0), tt, team)) return 0.0;
  team_sync<TT>(team);
  hermitian_part<NP, TT>(X, f, H, N, tt, S, team);
  team_tridiagonalize<NP, TT>(H, N, tt, S, team);
  for (int i = 0; i < N; ++i)
    if (!isfinite(S.d[i]) || (i + 1 < N && !isfinite(S.e2[i]))) return INFINITY;
  const double pivmin = tri_pivmin(S.e2, N);
  if (sturm_count(S.d, S.e2, N, -64.0 * N * eps * fmax(dmax, 1.0), pivmin) == 0) return 0.0;
  const double lmin = tri_eig(S.d, S.e2, N, 1), lmax = tri_eig(S.d, S.e2, N, N);
  const double bn = fmax(fabs(lmin), fabs(lmax));
  const double budget = 64.0 * N * eps * fmax(bn, 1.0);
  return fmax(0.0, fmax(0.0, -lmin) - budget) / fmax(bn, 2.2250738585072014e-308);
}

// Largest eigenvalue of the Hermitian H (destroyed); if `only_if_positive`,
// returns 0 without the multisection when no eigenvalue is >= 0.
template <int NP, int TT>
__device__ double team_lmax(Cx<double>* H, int N, int tt, ResScratch<NP>& S, int team, bool only_if_positive) {
  team_tridiagonalize<NP, TT>(H, N, tt, S, team);
  for (int i = 0; i < N; ++i)
    if (!isfinite(S.d[i]) || (i + 1 < N && !isfinite(S.e2[i]))) return INFINITY;
  if (only_if_positive && sturm_count(S.d, S.e2, N, 0.0, tri_pivmin(S.e2, N)) == N) return 0.0;
  return tri_eig(S.d, S.e2, N, N);
}

// The suite for N_b <= 16 and 17 ... 32 (residual_rows.cuh), in translation units of
// their own: a process loads a unit's kernels at the first launch of one of
// them (the first call of the suite in a process: 37 ms as one unit, 5 ms so).
template <typename RS> int launch_residual_rows_small(const ResidualArgs<RS>& a, cudaStream_t st);
template <typename RS> int launch_residual_rows_large(const ResidualArgs<RS>& a, cudaStream_t st);

}  // namespace qcl
