// Neighbour-period embedding self-energies: shifted sandwiches.
//
// Reference: _embedding_component_production / _embedding_self_energy_
// production (numerics/optimized/production_operators.jl:886-941); oracle
// embedding_self_energy (numerics/reference/periodicity.jl:113-150):
//   Sigma+^x(E) = T+ G^x(E + E^p) T+^H,  Sigma-^x(E) = T- G^x(E - E^p) T-^H,
// x in {R, <, >}, with G(E +- E^p) the 2-point linear interpolation of the
// EnergyShiftPlan and zero outside the window.
//
// One launch does all (sign, component) jobs, one per grid.z.  A CTA stages T
// and the blocks of BPC consecutive energies (interpolated on the way in) and
// multiplies in place: the product waits in registers until the tile has been
// read.  Bound by the latency of the scattered loads, so what counts is the
// number of resident warps and of loads in flight: one component per CTA and
// no second tile instead of three in turn with two.  N_b = 12, 400 x 16
// energies and momenta, complex128, both signs: 124 -> 92 us (177 MB, 27 us of
// HBM traffic); 8 energies per CTA: 8 us slower.
#include "blockmat.cuh"

namespace qcl {

template <typename R> struct SandwichArgs {
  int NE, Nk, N, njobs;
  SandwichJob jobs[2];
};

template <typename R, int NP, int BPC>
__device__ __forceinline__ void load_shifted(const Cx<R>* __restrict__ X, const ShiftPlanDev& plan, Cx<R>* bufs,
                                             int e0, int m, int NE, int Nk, int N) {
  // blockDim.x is a multiple of BPC, so each thread serves one energy of the
  // CTA: its interpolation plan is read once; the padded tile index is split
  // at compile time (entries past N are left as they are, as before)
  const int eloc = threadIdx.x % BPC;
  const int e = e0 + eloc;
  const bool ok = e < NE && plan.valid[e];
  int l = 0, r = 0;
  double th = 0.0;
  if (ok) {
    l = plan.left[e];
    r = plan.right[e];
    th = plan.theta[e];
  }
  const bool two = l != r && th != 0.0;
  const size_t base = (size_t)NE * m, cstride = (size_t)NE * Nk;
  constexpr int IT = NP * NP / Tile<NP>::TT, G = IT % 4 == 0 ? 4 : IT % 6 == 0 ? 6 : IT;  // elements in flight
  static_assert(IT * Tile<NP>::TT == NP * NP && IT % G == 0, "tile size");
  Cx<R>* dst = bufs + eloc * tile_stride<R, NP, BPC>();
#pragma unroll 1
  for (int q0 = 0; q0 < IT; q0 += G) {
    Cx<R> u[G], w[G];
#pragma unroll
    for (int q = 0; q < G; ++q) {
      const int el = (threadIdx.x + (q0 + q) * BPC * Tile<NP>::TT) / BPC, a = el % NP, b = el / NP;
      const size_t col = base + cstride * ((size_t)a + (size_t)N * b);
      const bool in = ok && a < N && b < N;
      u[q] = in ? X[col + l] : cx<R>(0, 0);
      w[q] = in && two ? X[col + r] : cx<R>(0, 0);
    }
#pragma unroll
    for (int q = 0; q < G; ++q) {
      const int el = (threadIdx.x + (q0 + q) * BPC * Tile<NP>::TT) / BPC;
      if (two) u[q] = cx<R>((R)((1 - th) * u[q].x + th * w[q].x), (R)((1 - th) * u[q].y + th * w[q].y));
      dst[sw<NP>(el % NP, el / NP)] = u[q];
    }
  }
}

// Registers are what limits the resident warps: 64 a thread where the
// accumulators leave room.
template <typename R, int NP, int BPC> constexpr int sandwich_min_ctas() {
  constexpr int regs = (NP >= 24 ? 80 : 64) * (sizeof(R) == 8 && NP >= 24 ? 2 : 1);
  return 65536 / (regs * BPC * Tile<NP>::TT);
}

template <typename R, int NP, int BPC>
__global__ void __launch_bounds__(BPC* Tile<NP>::TT, (sandwich_min_ctas<R, NP, BPC>())) sandwich_kernel(SandwichArgs<R> p) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t MSZ = tile_stride<R, NP, BPC>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<R>* Ts = reinterpret_cast<Cx<R>*>(smem_raw);
  Cx<R>* bufX = Ts + NP * NP;
  const int c = blockIdx.z % 3;
  const SandwichJob& job = p.jobs[blockIdx.z / 3];
  if (job.X[c] == nullptr || job.S[c] == nullptr) return;  // uniform
  const int N = p.N, NE = p.NE, Nk = p.Nk;
  const int m = blockIdx.y, e0 = blockIdx.x * BPC;
  const int team = threadIdx.x / TT, tt = threadIdx.x % TT;
  const Cx<double>* T = (const Cx<double>*)job.T;
  load_shifted<R, NP, BPC>((const Cx<R>*)job.X[c], job.plan, bufX, e0, m, NE, Nk, N);
  for (int i = threadIdx.x; i < NP * NP; i += blockDim.x) {
    const int a = i % NP, b = i / NP;
    Ts[sw<NP>(a, b)] = (a < N && b < N) ? cvt<R>(T[a + (size_t)N * b]) : cx<R>(0, 0);
  }
  Cx<R>* X = bufX + team * MSZ;
  __syncthreads();
  team_matmul_inplace<R, NP>(Ts, X, X, N, tt, team, false);  // X = T X
  team_matmul_inplace<R, NP>(X, Ts, X, N, tt, team, true);   // X = X T^H
  __syncthreads();
  store_blocks<R, R, NP, BPC>((Cx<R>*)job.S[c], bufX, MSZ, e0, m, NE, Nk, N);
}

template <typename R, int NP, int BPC>
static int launch_sandwich_t(const SandwichArgs<R>& a, cudaStream_t st) {
  constexpr int TT = Tile<NP>::TT;
  constexpr size_t smem = (NP * NP + BPC * tile_stride<R, NP, BPC>()) * sizeof(Cx<R>);
  static bool configured = false;
  if (!configured) {
    QCL_CUDA_CHECK(cudaFuncSetAttribute(sandwich_kernel<R, NP, BPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    configured = true;
  }
  dim3 grid((a.NE + BPC - 1) / BPC, a.Nk, 3 * a.njobs);
  sandwich_kernel<R, NP, BPC><<<grid, BPC * TT, smem, st>>>(a);
  QCL_LAUNCH_CHECK("sandwich_kernel");
  return QCL_OK;
}

template <typename R> static int launch_sandwich_p(const SandwichArgs<R>& a, cudaStream_t st) {
  constexpr bool wide = sizeof(R) == 8;
  switch (padded_size(a.N)) {
    case 8: return launch_sandwich_t<R, 8, 8>(a, st);
    case 16: return launch_sandwich_t<R, 16, wide ? 4 : 8>(a, st);
    case 24: return launch_sandwich_t<R, 24, 4>(a, st);
    case 32: return launch_sandwich_t<R, 32, wide ? 2 : 4>(a, st);
    case 48: return launch_sandwich_t<R, 48, 1>(a, st);
    default:
      set_last_error("basis size N_b=%d exceeds the supported maximum 48", a.N);
      return QCL_UNSUPPORTED;
  }
}

int launch_sandwich(int precision, int NE, int Nk, int N, const SandwichJob* jobs, int njobs, cudaStream_t st) {
  if (njobs < 1 || njobs > 2) {
    set_last_error("sandwich: 1 or 2 jobs per launch");
    return QCL_ARG;
  }
  if (precision == QCL_C128) {
    SandwichArgs<double> a;
    a.NE = NE; a.Nk = Nk; a.N = N; a.njobs = njobs;
    for (int j = 0; j < njobs; ++j) a.jobs[j] = jobs[j];
    return launch_sandwich_p<double>(a, st);
  }
  SandwichArgs<float> a;
  a.NE = NE; a.Nk = Nk; a.N = N; a.njobs = njobs;
  for (int j = 0; j < njobs; ++j) a.jobs[j] = jobs[j];
  return launch_sandwich_p<float>(a, st);
}

}  // namespace qcl
