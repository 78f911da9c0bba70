// Pointwise time-step operators and reductions (FP64): penalization, maximum
// velocity, per-case sums and the CFL time step.  Each kernel names the
// reference kernel it computes.
#include <algorithm>

#include "../../include/cup3d_b200.h"
#include "lab.cuh"
#include "stencils.cuh"
#include "profiler.h"

namespace cup3d {

struct Vec3 {
  double v[3];
};

// ---------------------------------------------------------------------------
// Penalization: KernelPenalization (Penalization.cpp:56-89) on obstacle blocks
// and the force/torque sums of kernelFinalizePenalizationForce (:91-109).
// ---------------------------------------------------------------------------
// In a batch (M.bcase set) each slot takes its case's kinematics and time
// step, and the force/torque sums go per slot into slot_force[6 * slot].
__global__ void __launch_bounds__(NT)
    k_penalize(DevMesh M, double* vel, const double* __restrict__ chi, ObstacleView ob, const double* __restrict__ kin,
               double dt, double lambda, int implicit, GridReduce G, double* force, double* slot_force) {
  __shared__ double red[8 * 6];
  const size_t n = size_t(M.nb) * BN;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int sl = blockIdx.x; sl < ob.nslots; sl += gridDim.x) {
    const int b = ob.blk[sl];
    const double* kn = M.case_kin ? M.case_kin + 9 * M.bcase[b] : kin;
    const double CM[3] = {kn[0], kn[1], kn[2]};
    const double V[3] = {kn[3], kn[4], kn[5]};
    const double O[3] = {kn[6], kn[7], kn[8]};
    const double dtb = block_dt(M, b, dt);
    const double lambdaFac = implicit ? lambda : 1.0 / dtb;
    const double h = M.h[b], dv = h * h * h;
    for (int cell = threadIdx.x; cell < BN; cell += NT) {
      const size_t gi = size_t(b) * BN + cell;
      const double CHI = ob.chi[size_t(sl) * BN + cell];
      if (chi[gi] > CHI) continue;
      if (CHI <= 0) continue;
      const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
      double p[3] = {(M.index[3 * b] * BS + x + 0.5) * h, (M.index[3 * b + 1] * BS + y + 0.5) * h,
                     (M.index[3 * b + 2] * BS + z + 0.5) * h};
      p[0] -= CM[0];
      p[1] -= CM[1];
      p[2] -= CM[2];
      const double* ud = ob.udef;
      const size_t ns = ob.nslots;
      const double U0 = V[0] + O[1] * p[2] - O[2] * p[1] + ud[(0 * ns + sl) * BN + cell];
      const double U1 = V[1] + O[2] * p[0] - O[0] * p[2] + ud[(1 * ns + sl) * BN + cell];
      const double U2 = V[2] + O[0] * p[1] - O[1] * p[0] + ud[(2 * ns + sl) * BN + cell];
      const double X = implicit ? (CHI > 0.5 ? 1.0 : 0.0) : CHI;
      const double penalFac = implicit ? X * lambdaFac / (1 + X * lambdaFac * dtb) : X * lambdaFac;
      const double FPX = penalFac * (U0 - vel[gi]);
      const double FPY = penalFac * (U1 - vel[n + gi]);
      const double FPZ = penalFac * (U2 - vel[2 * n + gi]);
      vel[gi] = vel[gi] + dtb * FPX;
      vel[n + gi] = vel[n + gi] + dtb * FPY;
      vel[2 * n + gi] = vel[2 * n + gi] + dtb * FPZ;
      acc[0] += dv * FPX;
      acc[1] += dv * FPY;
      acc[2] += dv * FPZ;
      acc[3] += dv * (p[1] * FPZ - p[2] * FPY);
      acc[4] += dv * (p[2] * FPX - p[0] * FPZ);
      acc[5] += dv * (p[0] * FPY - p[1] * FPX);
    }
    if (slot_force) {  // uniform over the CTA
      block_reduce<6>(acc, red);
      if (threadIdx.x == 0)
        for (int q = 0; q < 6; ++q) slot_force[6 * sl + q] = acc[q];
      for (int q = 0; q < 6; ++q) acc[q] = 0.0;
    }
  }
  if (!slot_force && grid_reduce<6>(acc, G, red) && threadIdx.x == 0)
    for (int q = 0; q < 6; ++q) force[q] = acc[q];
}

int launch_penalize(const DevMesh& M, double* vel, const double* chi, const ObstacleView& ob, const double* kin,
                    double dt, double lambda, int implicit, double* force, double* partial, unsigned* counter,
                    cudaStream_t s, double* slot_force) {
  if (ob.nslots <= 0) {
    if (slot_force) return 0;
    CUP_CUDA_TRY(cudaMemsetAsync(force, 0, 6 * sizeof(double), s));
    return 0;
  }
  const int grid = std::min(ob.nslots, 1184);
  GridReduce G{partial, counter};
  ProfScope ps("penalize", s);
  k_penalize<<<grid, NT, 0, s>>>(M, vel, chi, ob, kin, dt, lambda, implicit, G, force, slot_force);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// findMaxU (ProcessHelpers.h:71-94)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) k_max_u(size_t n, const double* __restrict__ vel, Vec3 ui, GridReduce G,
                                              double* out) {
  __shared__ double red[8];
  double m = 0.0;
  for (size_t i = size_t(blockIdx.x) * NT + threadIdx.x; i < n; i += size_t(gridDim.x) * NT) {
    const double a = fabs(vel[i] + ui.v[0]);
    const double b = fabs(vel[n + i] + ui.v[1]);
    const double c = fabs(vel[2 * n + i] + ui.v[2]);
    m = fmax(m, fmax(a, fmax(b, c)));
  }
  if (grid_reduce_max(m, G, red) && threadIdx.x == 0) *out = m;
}

int launch_max_u(const DevMesh& M, const double* vel, const double* uinf, double* out, double* partial,
                 unsigned* counter, int grid, cudaStream_t s) {
  GridReduce G{partial, counter};
  Vec3 ui{{uinf[0], uinf[1], uinf[2]}};
  ProfScope ps("max_u", s);
  k_max_u<<<grid, NT, 0, s>>>(size_t(M.nb) * BN, vel, ui, G, out);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// Per-case reductions of a batch: per-item values (blocks or obstacle slots),
// then one CTA per case over the case's item range, in a fixed order.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) k_block_max_u(DevMesh M, const double* __restrict__ vel, Vec3 ui,
                                                    double* bmax) {
  __shared__ double red[NT / 32];
  const size_t n = size_t(M.nb) * BN;
  for (int b = blockIdx.x; b < M.nb; b += gridDim.x) {
    double m = 0.0;
    for (int c = threadIdx.x; c < BN; c += NT) {
      const size_t i = size_t(b) * BN + c;
      m = fmax(m, fmax(fabs(vel[i] + ui.v[0]), fmax(fabs(vel[n + i] + ui.v[1]), fabs(vel[2 * n + i] + ui.v[2]))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      double mm = 0.0;
      for (int w = 0; w < NT / 32; ++w) mm = fmax(mm, red[w]);
      bmax[b] = mm;
    }
  }
}

// (sum phi h^3, sum h^3) of each block
__global__ void __launch_bounds__(NT) k_block_sums(DevMesh M, const double* __restrict__ phi, double* bsum) {
  __shared__ double red[64];
  for (int b = blockIdx.x; b < M.nb; b += gridDim.x) {
    const double h = M.h[b], h3 = h * h * h;
    double v[1] = {0.0};
    for (int c = threadIdx.x; c < BN; c += NT) v[0] += phi[size_t(b) * BN + c];
    block_reduce<1>(v, red);
    if (threadIdx.x == 0) {
      bsum[2 * b] = v[0] * h3;
      bsum[2 * b + 1] = BN * h3;
    }
  }
}

// out[NR c + r] = sum (MAX = 0) or max (MAX = 1) of in[NR i + r], i in [first[c], first[c+1])
template <int NR, int MAX>
__global__ void __launch_bounds__(NT) k_case_reduce(const double* __restrict__ in, const int* __restrict__ first,
                                                    double* out) {
  __shared__ double red[8 * NR];
  const int c = blockIdx.x;
  double v[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) v[r] = 0.0;
  for (int i = first[c] + threadIdx.x; i < first[c + 1]; i += NT)
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = MAX ? fmax(v[r], in[size_t(NR) * i + r]) : v[r] + in[size_t(NR) * i + r];
  if (MAX) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[r] = fmax(v[r], __shfl_xor_sync(0xffffffffu, v[r], o));
      if ((threadIdx.x & 31) == 0) red[(threadIdx.x >> 5) * NR + r] = v[r];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int r = 0; r < NR; ++r) {
        double m = 0.0;
        for (int w = 0; w < NT / 32; ++w) m = fmax(m, red[w * NR + r]);
        out[NR * c + r] = m;
      }
  } else {
    block_reduce<NR>(v, red);
    if (threadIdx.x == 0)
      for (int r = 0; r < NR; ++r) out[NR * c + r] = v[r];
  }
}

int launch_case_max_u(const DevMesh& M, const double* vel, const double* uinf, double* bmax, const int* first,
                      int ncase, double* out, int grid, cudaStream_t s) {
  Vec3 ui{{uinf[0], uinf[1], uinf[2]}};
  ProfScope ps("case_max_u", s);
  k_block_max_u<<<grid, NT, 0, s>>>(M, vel, ui, bmax);
  k_case_reduce<1, 1><<<ncase, NT, 0, s>>>(bmax, first, out);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

int launch_case_sums(const DevMesh& M, const double* phi, double* bsum, const int* first, int ncase, double* out,
                     int grid, cudaStream_t s) {
  ProfScope ps("case_sums", s);
  k_block_sums<<<grid, NT, 0, s>>>(M, phi, bsum);
  k_case_reduce<2, 0><<<ncase, NT, 0, s>>>(bsum, first, out);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

int launch_case_forces(const double* slot_force, const int* slot_first, int ncase, double* out, cudaStream_t s) {
  ProfScope ps("case_forces", s);
  k_case_reduce<6, 0><<<ncase, NT, 0, s>>>(slot_force, slot_first, out);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// Simulation::calcMaxTimestep on the device, for captured steps: the same
// operations in the same order as the host version (no contraction), with
// the CFL factor (ramped or not) computed on the host: bit-identical dt.
// ---------------------------------------------------------------------------
__global__ void k_calc_dt(const double* __restrict__ umax, const double* __restrict__ cfl_fac, double nu,
                          double hmin, double* dt) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double u = *umax;
  const double t = __dmul_rn(1.0 / 6.0, hmin);
  const double dtDiffusion = __ddiv_rn(__dmul_rn(t, hmin), __dadd_rn(nu, __dmul_rn(t, u)));
  const double dtAdvection = __ddiv_rn(hmin, __dadd_rn(u, 1e-8));
  const double cand = __dmul_rn(*cfl_fac, dtAdvection);
  *dt = cand < dtDiffusion ? cand : dtDiffusion;
}

int launch_calc_dt(const double* umax, const double* cfl_fac, double nu, double hmin, double* dt, cudaStream_t s) {
  k_calc_dt<<<1, 32, 0, s>>>(umax, cfl_fac, nu, hmin, dt);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// The same per case of a batch: dt[c] from umax[c] and hmin[c].
__global__ void k_case_calc_dt(const double* __restrict__ umax, const double* __restrict__ cfl_fac, double nu,
                               const double* __restrict__ hmin, int ncase, double* dt) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncase) return;
  const double u = umax[c], hm = hmin[c];
  const double t = __dmul_rn(1.0 / 6.0, hm);
  const double dtDiffusion = __ddiv_rn(__dmul_rn(t, hm), __dadd_rn(nu, __dmul_rn(t, u)));
  const double dtAdvection = __ddiv_rn(hm, __dadd_rn(u, 1e-8));
  const double cand = __dmul_rn(*cfl_fac, dtAdvection);
  dt[c] = cand < dtDiffusion ? cand : dtDiffusion;
}

int launch_case_calc_dt(const double* umax, const double* cfl_fac, double nu, const double* hmin, int ncase,
                        double* dt, cudaStream_t s) {
  k_case_calc_dt<<<(ncase + 127) / 128, 128, 0, s>>>(umax, cfl_fac, nu, hmin, ncase, dt);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace cup3d
