// Current and population reductions (FP64, fixed-order).
//
// Current (_production_boundary_flux_bar, numerics/optimized/production_
// iteration.jl:174-201; oracle _boundary_flux_complex, physics/observables.jl:
// 176-214):
//   Jbar = Re[ g_s/(2 pi) sum_{e,m} wE_e wk_m sum_{a,b}
//              (S>_{em,ab} G<_{em,ba} - S<_{em,ab} G>_{em,ba}) ]
// Populations (_production_state_populations, production_iteration.jl:
// 204-215):  p_a = Re[-i g_s/(2 pi) sum_{e,m} wE wk G<_{em,aa}] / target.
//
// The reference accumulates the current in (|eps|, eps) order to limit
// cancellation; here every term is accumulated in FP64 by a fixed two-level
// tree (per-thread strided sums, fixed CTA partials combined in CTA order),
// which is deterministic and whose rounding is of the same order.
#include "kernels.cuh"

namespace qcl {

constexpr int OBS_CTAS = 296, OBS_THREADS = 256;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int K> __device__ __forceinline__ void cta_sum(double (&v)[K], double* out) {
  __shared__ double red[K][OBS_THREADS / 32];
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = wsum(v[k]);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) red[k][threadIdx.x >> 5] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double s = 0;
      for (int w = 0; w < OBS_THREADS / 32; ++w) s += red[k][w];
      out[k] = s;
    }
}

// One launch.  A CTA owns 256 consecutive (e, m): each thread's weight is read
// once, every field access is contiguous, and the CTAs of a row of the grid
// take slices of the (a, b) of the current (blockIdx.y < S) or the diagonal
// of the populations (blockIdx.y = S).  The CTA that finishes last adds the
// partial sums in CTA order:
//   out[0] = Jbar, out[1] = Im of the complex flux (diagnostic),
//   out[2 + a] = p_a.
// Bound by the four field reads: 537 MB at N_E x N_k = 1024 x 32, N_b = 16,
// complex128: 139 + 10 + 4 us in three launches with a division per element -> 94 us.
constexpr int OBS_SLICES = 8;
template <typename R>
__global__ void __launch_bounds__(OBS_THREADS)
    observables_kernel(int NE, int Nk, int N, const double* __restrict__ wE, const double* __restrict__ wk,
                       const Cx<R>* __restrict__ SG, const Cx<R>* __restrict__ SL, const Cx<R>* __restrict__ GL,
                       const Cx<R>* __restrict__ GG, int gs, double target, double* partial, unsigned* counter,
                       double* out) {
  const long long blocks = (long long)NE * Nk;
  const int S = (int)gridDim.y - 1;
  double* cur = partial;                                         // [gridDim.x][S][2]
  double* pop = partial + 2 * (size_t)gridDim.x * OBS_SLICES;   // [N][gridDim.x][2]
  const long long step = (long long)gridDim.x * OBS_THREADS;
  if ((int)blockIdx.y < S) {
    const int q0 = N * N * blockIdx.y / S, q1 = N * N * (blockIdx.y + 1) / S;
    double v[2] = {0, 0};
    for (long long em = blockIdx.x * (long long)OBS_THREADS + threadIdx.x; em < blocks; em += step) {
      const double w = wE[em % NE] * wk[em / NE];
      double re = 0, im = 0;
      int a = q0 % N, b = q0 / N;
#pragma unroll 4
      for (int q = q0; q < q1; ++q) {
        const size_t i = (size_t)em + (size_t)blocks * q, it = (size_t)em + (size_t)blocks * (b + N * a);
        const Cx<R> sg = SG[i], sl = SL[i], gl = GL[it], gg = GG[it];
        re += ((double)sg.x * gl.x - (double)sg.y * gl.y) - ((double)sl.x * gg.x - (double)sl.y * gg.y);
        im += ((double)sg.x * gl.y + (double)sg.y * gl.x) - ((double)sl.x * gg.y + (double)sl.y * gg.x);
        if (++a == N) {
          a = 0;
          ++b;
        }
      }
      v[0] += w * re;
      v[1] += w * im;
    }
    cta_sum<2>(v, cur + 2 * ((size_t)blockIdx.x * S + blockIdx.y));
  } else {
    for (int a = 0; a < N; ++a) {
      double v[2] = {0, 0};
      for (long long em = blockIdx.x * (long long)OBS_THREADS + threadIdx.x; em < blocks; em += step) {
        const Cx<R> g = GL[(size_t)em + (size_t)blocks * (a + N * a)];
        const double w = wE[em % NE] * wk[em / NE];
        v[0] += w * g.x;
        v[1] += w * g.y;
      }
      cta_sum<2>(v, pop + 2 * ((size_t)a * gridDim.x + blockIdx.x));
      __syncthreads();  // the sum's scratch is reused
    }
  }
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1u) == gridDim.x * gridDim.y - 1;
    if (last) *counter = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const double pre = gs / (2.0 * M_PI);
  for (int q = threadIdx.x >> 5; q < 1 + N; q += OBS_THREADS / 32) {  // one warp per quantity
    const double* src = q == 0 ? cur : pop + 2 * (size_t)(q - 1) * gridDim.x;
    const int count = q == 0 ? (int)gridDim.x * S : (int)gridDim.x;
    double re = 0, im = 0;
    for (int c = threadIdx.x & 31; c < count; c += 32) {
      re += __ldcg(src + 2 * c);
      im += __ldcg(src + 2 * c + 1);
    }
    re = wsum(re);
    im = wsum(im);
    if ((threadIdx.x & 31) != 0) continue;
    if (q == 0) {
      out[0] = pre * re;
      out[1] = pre * im;
    } else {
      out[1 + q] = pre * im / target;  // -i pre (re + i im) = pre (im - i re): real part = pre * im
    }
  }
}

size_t observables_partial_doubles(int N) { return 2 * (size_t)OBS_CTAS * (OBS_SLICES + N) + 1; }

// SG, SL: the plus-embedding family (Sigma+^>, Sigma+^<); GL, GG: the state.
// partial: observables_partial_doubles(N), of which the last is the CTA
// counter, zero before the first launch.
int launch_observables(int precision, int NE, int Nk, int N, const double* wE, const double* wk, const void* SG,
                       const void* SL, const void* GL, const void* GG, int gs, double target, double* partial,
                       double* out, cudaStream_t st) {
  const long long g = ((long long)NE * Nk + OBS_THREADS - 1) / OBS_THREADS;
  const dim3 grid((unsigned)(g < OBS_CTAS ? g : OBS_CTAS), (N * N < OBS_SLICES ? N * N : OBS_SLICES) + 1);
  unsigned* counter = (unsigned*)(partial + observables_partial_doubles(N) - 1);
  if (precision == QCL_C128)
    observables_kernel<double><<<grid, OBS_THREADS, 0, st>>>(NE, Nk, N, wE, wk, (const Cx<double>*)SG,
                                                             (const Cx<double>*)SL, (const Cx<double>*)GL,
                                                             (const Cx<double>*)GG, gs, target, partial, counter, out);
  else
    observables_kernel<float><<<grid, OBS_THREADS, 0, st>>>(NE, Nk, N, wE, wk, (const Cx<float>*)SG,
                                                            (const Cx<float>*)SL, (const Cx<float>*)GL,
                                                            (const Cx<float>*)GG, gs, target, partial, counter, out);
  QCL_LAUNCH_CHECK("observables");
  return QCL_OK;
}

}  // namespace qcl
