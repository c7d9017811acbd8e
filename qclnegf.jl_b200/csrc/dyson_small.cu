#include "dyson.cuh"

namespace qcl {

// A magnitude's bits as one integer, for exact comparisons, and the test for
// zero of the warp-per-block kernel's keys (dyson.cu).
__device__ __forceinline__ unsigned long long mag_bits(double mag) { return (unsigned long long)__double_as_longlong(mag); }
__device__ __forceinline__ unsigned mag_bits(float mag) { return __float_as_uint(mag); }
__device__ __forceinline__ bool mag_zero(unsigned long long bits) { return (bits >> 38) == 0u; }
__device__ __forceinline__ bool mag_zero(unsigned bits) { return (bits >> 6) == 0u; }

// ---------------------------------------------------------------------------
// Small bases (N_b <= 6): one thread per (E, k) block, the block in registers.
// The lanes of a warp are 32 consecutive energies, so every element of a field
// is one contiguous access of the warp and nothing goes through shared memory; a warp-per-block team pads N_b = 5
// to 8 x 8 and works with 20 of 32 lanes.  In-place Gauss-Jordan with row
// interchanges (predicated swaps keep every register index static), then the
// products row by row with Sigma re-read from L1 (a second N x N register
// block would spill).  Bound by FP64 issue and load latency at 8 warps per SM.
// N_E x N_k = 2401 x 61, complex128, G^R, G^<, G^>: N_b = 5 696 -> 131 us (54 us
// of HBM traffic), N_b = 3 569 -> 35 us, N_b = 6 733 -> 238 us.
// ---------------------------------------------------------------------------
constexpr int kSmallThreads = 64;

template <typename RS, typename RL, typename RM, int N>
__global__ void __launch_bounds__(kSmallThreads) dyson_small_kernel(DysonArgs<RS> p) {
  const int e = blockIdx.x * kSmallThreads + threadIdx.x, NE = p.NE, Nk = p.Nk, m = p.m0 + blockIdx.y;
  if (e >= NE) return;
  const size_t at = (size_t)e + (size_t)NE * m, cs = (size_t)NE * Nk;
  Cx<RL> w[N][N];
  const double eps_e = p.eps[e];
  double s = 0.0;
#pragma unroll
  for (int a = 0; a < N; ++a) {
    double rsum = 0.0;
#pragma unroll
    for (int b = 0; b < N; ++b) {
      const Cx<double> hv = p.h[(size_t)m + (size_t)Nk * (a + N * b)];
      const Cx<RS> sv = p.sigR[at + cs * (a + N * b)];
      double re = -hv.x - (double)sv.x, im = -hv.y - (double)sv.y;
      if (a == b) {
        re += eps_e;
        im += p.eta;
      }
      w[a][b] = cx<RL>((RL)re, (RL)im);
      rsum += sqrt(re * re + im * im);
    }
    s = fmax(s, rsum);
  }
  const RL inv_s = (RL)(1.0 / s);
  const bool scale_ok = s > 0.0 && isfinite(s);
#pragma unroll
  for (int a = 0; a < N; ++a)
#pragma unroll
    for (int b = 0; b < N; ++b) w[a][b] = inv_s * w[a][b];
  int piv[N], zstep = -1;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    // by the bits of the magnitudes, as the keys are: a NaN ranks above any number
    int best = k;
    auto mag = mag_bits(cabs1(w[k][k]));
#pragma unroll
    for (int r = k + 1; r < N; ++r) {
      const auto q = mag_bits(cabs1(w[r][k]));
      if (q > mag) {
        mag = q;
        best = r;
      }
    }
    piv[k] = best;
    const bool zero = mag_zero(mag);
    if (zero && zstep < 0) zstep = k;
#pragma unroll
    for (int r = k + 1; r < N; ++r)
#pragma unroll
      for (int b = 0; b < N; ++b) {
        const Cx<RL> x = w[k][b], y = w[r][b];
        w[k][b] = best == r ? y : x;
        w[r][b] = best == r ? x : y;
      }
    const Cx<RL> rp = zero ? cx<RL>(0, 0) : crecip_pivot(w[k][k]);
    w[k][k] = cx<RL>(1, 0);
#pragma unroll
    for (int b = 0; b < N; ++b) w[k][b] = rp * w[k][b];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      if (r == k) continue;
      const Cx<RL> f = w[r][k];
      w[r][k] = cx<RL>(0, 0);
#pragma unroll
      for (int b = 0; b < N; ++b) cfms(w[r][b], f, w[k][b]);
    }
  }
#pragma unroll
  for (int k = N - 1; k >= 0; --k)  // undo the interchanges on the columns
#pragma unroll
    for (int c = k + 1; c < N; ++c)
#pragma unroll
      for (int a = 0; a < N; ++a) {
        const Cx<RL> x = w[a][k], y = w[a][c];
        w[a][k] = piv[k] == c ? y : x;
        w[a][c] = piv[k] == c ? x : y;
      }
  if (!scale_ok || zstep >= 0)
    record_status(p.status, QCL_SINGULAR, (long long)at * kSingularPivotSpan + (scale_ok ? zstep + 1 : 0));
  if (p.scale) p.scale[at] = s;
  Cx<RS> g[N][N];
#pragma unroll
  for (int a = 0; a < N; ++a)
#pragma unroll
    for (int b = 0; b < N; ++b) {
      g[a][b] = cvt<RS>(inv_s * w[a][b]);
      if (p.GR) p.GR[at + cs * (a + N * b)] = g[a][b];
    }
#pragma unroll 1
  for (int which = 0; which < 2; ++which) {
    const Cx<RS>* __restrict__ sig = which == 0 ? p.sigL : p.sigG;
    Cx<RS>* __restrict__ out = which == 0 ? p.GL : p.GG;
    Cx<double>* tr = which == 0 ? p.traceL : p.traceG;
    if (sig == nullptr || out == nullptr) continue;
    double tre = 0, tim = 0;
#pragma unroll
    for (int a = 0; a < N; ++a) {
      Cx<RM> t[N];
#pragma unroll
      for (int b = 0; b < N; ++b) t[b] = cx<RM>(0, 0);
#pragma unroll
      for (int l = 0; l < N; ++l)
#pragma unroll
        for (int b = 0; b < N; ++b) cfma(t[b], cvt<RM>(g[a][l]), cvt<RM>(sig[at + cs * (l + N * b)]));
#pragma unroll
      for (int b = 0; b < N; ++b) {
        const Cx<RS> tb = cvt<RS>(t[b]);  // the product is stored between the two stages, as in the team kernel
        t[b] = cvt<RM>(tb);
      }
#pragma unroll
      for (int b = 0; b < N; ++b) {
        Cx<RM> o = cx<RM>(0, 0);
#pragma unroll
        for (int l = 0; l < N; ++l) cfma_conj(o, t[l], cvt<RM>(g[b][l]));
        const Cx<RS> v = cvt<RS>(o);
        out[at + cs * (a + N * b)] = v;
        if (a == b) {
          tre += (double)v.x;
          tim += (double)v.y;
        }
      }
    }
    if (tr) tr[at] = cx<double>(tre, tim);
  }
}

template <typename RS, typename RL, typename RM>
int launch_dyson_small(const DysonArgs<RS>& a, cudaStream_t st) {
  const dim3 grid((a.NE + kSmallThreads - 1) / kSmallThreads, a.mcount);
#define SMALL(NV) \
  case NV: dyson_small_kernel<RS, RL, RM, NV><<<grid, kSmallThreads, 0, st>>>(a); break
  switch (a.N) {
    SMALL(1);
    SMALL(2);
    SMALL(3);
    SMALL(4);
    SMALL(5);
    SMALL(6);
  }
#undef SMALL
  QCL_LAUNCH_CHECK("dyson_small_kernel");
  return QCL_OK;
}
template int launch_dyson_small<double, double, double>(const DysonArgs<double>&, cudaStream_t);
template int launch_dyson_small<float, double, float>(const DysonArgs<float>&, cudaStream_t);
template int launch_dyson_small<float, float, float>(const DysonArgs<float>&, cudaStream_t);

}  // namespace qcl
