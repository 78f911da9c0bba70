// Time-step stencil operators (FP64), one CTA per 8^3 block with its ghost
// layers staged in shared memory.  Each kernel names the reference kernel it
// computes; coarse-fine flux correction (Cubism FluxCorrection, absent from the
// reference tree) adds, to a coarse cell next to a finer face, its own face
// value plus the four fine face values, computed by the coarse block's CTA
// from the fine blocks' face cells and their ghosts.
#include <algorithm>

#include "../../include/cup3d_b200.h"
#include "lab.cuh"
#include "staged.cuh"
#include "stencils.cuh"
#include "profiler.h"

namespace cup3d {

struct Vec3 {
  double v[3];
};

// lab coordinates of own face cell (layer 0) and the ghost at layer 1
__device__ __forceinline__ void face_lab_pair(int d, int s, int a, int bb, int q[3], int g[3]) {
  q[d] = s ? BS - 1 : 0;
  q[tan1(d)] = a;
  q[tan2(d)] = bb;
  g[0] = q[0];
  g[1] = q[1];
  g[2] = q[2];
  g[d] += s ? 1 : -1;
}

// ---------------------------------------------------------------------------
// PressureProjection RHS: KernelPressureRHS (PressureProjection.cpp:96-199),
// kernelUpdateTmpV (:202-242) and KernelDivPressure (:16-94, step > 2).
// ---------------------------------------------------------------------------
struct UdefGet {
  ObstacleView ob;
  const double* chi;
  __device__ __forceinline__ double operator()(int c, int blk, int cell) const {
    const int sl = ob.slot[blk];
    if (sl < 0) return 0.0;
    return chi[size_t(blk) * BN + cell] <= ob.chi[size_t(sl) * BN + cell]
               ? ob.udef[(size_t(c) * ob.nslots + sl) * BN + cell]
               : 0.0;
  }
};

// One CTA walks its blocks through the staged pipeline (staged.cuh): the
// velocity and p_old labs arrive by bulk copies and per-cell async copies
// while the previous block is computed.  Blocks next to the body (rare) add
// the u_def lab with plain loads.
template <int USE_POLD>
__global__ void __launch_bounds__(NT, 2)
    k_pressure_rhs(DevMesh M, const double* __restrict__ vel, const double* __restrict__ pold,
                   const double* __restrict__ chi, ObstacleView ob, double dt, double* __restrict__ lhs,
                   double* __restrict__ phi) {
  extern __shared__ __align__(16) unsigned char stage_smem[];
  constexpr int NCH = 3 + USE_POLD;
  using SS = StagedShape<NCH, 0>;
  using LG = LabGeom<1>;
  double* dlab = reinterpret_cast<double*>(stage_smem + SS::kBytes);
  double* corr = dlab + 3 * LG::V;  // [0,512): RHS flux correction, [512,1024): div p correction
  const size_t n = size_t(M.nb) * BN;
  const double* src[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) src[c] = c < 3 ? vel + c * n : pold;
  auto getV = [&](int c, int blk, int cell) { return vel[c * n + size_t(blk) * BN + cell]; };
  auto getP = [&](int, int blk, int cell) { return pold[size_t(blk) * BN + cell]; };
  UdefGet getD{ob, chi};
  staged_blocks<NCH, 0>(M, src, ob.near, stage_smem, M.kerr, [&](int, int b, const StageMeta& m, double* ulab) {
    double* plab = ulab + 3 * LG::V;
    stage_fixup<3>(ulab, M, m, getV, true);
    if (USE_POLD) stage_fixup<1>(plab, M, m, getP, false);
    const bool near = m.flag != 0;
    if (near) lab_fill<1, 3>(dlab, M, b, getD, true);
    const bool fix = meta_has_finer(m);
    if (fix)
      for (int i = threadIdx.x; i < 2 * BN; i += NT) corr[i] = 0.0;
    __syncthreads();
    const double dtb = block_dt(M, b, dt);
    const double h = m.h, fac = 0.5 * h * h / dtb;
    auto U = [&](int c, int x, int y, int z) { return ulab[c * LG::V + LG::at(x, y, z)]; };
    auto D = [&](int c, int x, int y, int z) { return near ? dlab[c * LG::V + LG::at(x, y, z)] : 0.0; };
    auto P = [&](int x, int y, int z) { return plab[LG::at(x, y, z)]; };
    if (fix) {
      for (int f = 0; f < 6; ++f) {
        if (m.kind[f] != K_FINER) continue;
        const int d = f >> 1, s = f & 1;
        if (threadIdx.x < 64) {
          const int a = threadIdx.x & 7, bb = threadIdx.x >> 3;
          int q[3], g[3];
          face_lab_pair(d, s, a, bb, q, g);
          const int ch = m.nbr[4 * f + (a >> 2) + 2 * (bb >> 2)];
          const double hf = M.h[ch], facf = 0.5 * hf * hf / dtb;
          const int oc = face_cell(d, s, 0, a, bb);
          const double sg = s ? -1.0 : 1.0, sgc = -sg;
          const double cq = chi[size_t(b) * BN + oc];
          double vr = sg * fac * (U(d, g[0], g[1], g[2]) + U(d, q[0], q[1], q[2])) -
                      sg * cq * fac * (D(d, g[0], g[1], g[2]) + D(d, q[0], q[1], q[2]));
          double vp = USE_POLD ? h * (P(q[0], q[1], q[2]) - P(g[0], g[1], g[2])) : 0.0;
#pragma unroll
          for (int e2 = 0; e2 < 2; ++e2)
#pragma unroll
            for (int e1 = 0; e1 < 2; ++e1) {
              const int fa = 2 * (a & 3) + e1, fb = 2 * (bb & 3) + e2;
              const int cf = face_cell(d, 1 - s, 0, fa, fb);
              const double uf = getV(d, ch, cf);
              const double gu = child_ghost1([&](int cell) { return getV(d, b, cell); }, M, ch, d, s, fa, fb);
              const double cf_chi = chi[size_t(ch) * BN + cf];
              double df = 0.0, gd = 0.0;
              if (near) {
                df = getD(d, ch, cf);
                gd = child_ghost1([&](int cell) { return getD(d, b, cell); }, M, ch, d, s, fa, fb);
              }
              vr += sgc * facf * (gu + uf) - sgc * cf_chi * facf * (gd + df);
              if (USE_POLD) {
                const double pf = getP(0, ch, cf);
                const double gp = child_ghost1([&](int cell) { return getP(0, b, cell); }, M, ch, d, s, fa, fb);
                vp += hf * (pf - gp);
              }
            }
          corr[oc] += vr;
          corr[BN + oc] += vp;
        }
        __syncthreads();
      }
    }
    for (int qq = 0; qq < 2; ++qq) {
      const int cell = threadIdx.x + qq * NT;
      const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
      const size_t gi = size_t(b) * BN + cell;
      double p = fac * (U(0, x + 1, y, z) - U(0, x - 1, y, z) + U(1, x, y + 1, z) - U(1, x, y - 1, z) +
                        U(2, x, y, z + 1) - U(2, x, y, z - 1));
      if (near) {
        const double divUs = D(0, x + 1, y, z) - D(0, x - 1, y, z) + D(1, x, y + 1, z) - D(1, x, y - 1, z) +
                             D(2, x, y, z + 1) - D(2, x, y, z - 1);
        p += -chi[gi] * fac * divUs;
      }
      if (fix) p += corr[cell];
      if (USE_POLD) {
        double dp = h * (P(x + 1, y, z) + P(x - 1, y, z) + P(x, y + 1, z) + P(x, y - 1, z) + P(x, y, z + 1) +
                         P(x, y, z - 1) - 6.0 * P(x, y, z));
        if (fix) dp += corr[BN + cell];
        p -= dp;
      }
      lhs[gi] = p;
      phi[gi] = 0.0;
    }
    __syncthreads();
  });
}

// CTAs of a staged kernel that fit on the device at once: the pipeline wants
// one resident wave of CTAs, each walking several blocks.
template <class K>
static int resident_ctas(K kern, size_t smem, unsigned long long& cached_mask, int* cache) {
  int dev = 0;
  CUP_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev > 63) return set_error(CUP_ERR_ARG, "device ordinal above 63");
  if (first_on_device(cached_mask)) {
    int per_sm = 0, sms = 0;
    CUP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    CUP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem));
    CUP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (per_sm < 1) return set_error(CUP_ERR_CUDA, "staged stencil kernel does not fit on an SM");
    cache[dev] = per_sm * sms;
  }
  return 0;
}

template <int USE_POLD>
constexpr size_t rhs_smem() {
  return StagedShape<3 + USE_POLD, 0>::kBytes + (3 * LabGeom<1>::V + 2 * BN) * sizeof(double);
}

int launch_pressure_rhs(const DevMesh& M, const double* vel, const double* pold, const double* chi,
                        const ObstacleView& ob, double dt, int step, int step_2nd_start, double* lhs, double* phi,
                        int grid, cudaStream_t s) {
  static unsigned long long attr[2] = {0, 0};
  static int resident[2][64];
  int dev = 0;
  CUP_CUDA_TRY(cudaGetDevice(&dev));
  ProfScope ps("pressure_rhs", s);
  // with udef = 0 in every slot the near-body terms (chi times the
  // divergence of udef, with its flux correction) are exact zeros: no block
  // needs the udef lab
  ObstacleView o = ob;
  if (o.udef_zero) o.near = nullptr;
  if (step > step_2nd_start) {
    if (int rc = resident_ctas(k_pressure_rhs<1>, rhs_smem<1>(), attr[1], resident[1])) return rc;
    grid = std::max(1, std::min({grid, resident[1][dev], M.nb}));
    k_pressure_rhs<1><<<grid, NT, rhs_smem<1>(), s>>>(M, vel, pold, chi, o, dt, lhs, phi);
  } else {
    if (int rc = resident_ctas(k_pressure_rhs<0>, rhs_smem<0>(), attr[0], resident[0])) return rc;
    grid = std::max(1, std::min({grid, resident[0][dev], M.nb}));
    k_pressure_rhs<0><<<grid, NT, rhs_smem<0>(), s>>>(M, vel, pold, chi, o, dt, lhs, phi);
  }
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// Mean removal + incremental pressure (PressureProjection.cpp:404-446) fused
// with KernelGradP (:244-323) and the velocity update (:451-467).  The
// pressure p = phi - avg (+ p_old) is formed at the point of use from the
// staged phi and p_old labs; the velocity comes in with them as interiors.
// ---------------------------------------------------------------------------
template <int USE_POLD>
__global__ void __launch_bounds__(NT, 3)
    k_grad_update(DevMesh M, double* vel, const double* __restrict__ phi, const double* __restrict__ pold,
                  double* __restrict__ pnew, const double* sums, double dt) {
  extern __shared__ __align__(16) unsigned char stage_smem[];
  constexpr int NCH = 1 + USE_POLD;
  using SS = StagedShape<NCH, 3>;
  using LG = LabGeom<1>;
  double* corr = reinterpret_cast<double*>(stage_smem + SS::kBytes);  // 3 BN
  const size_t n = size_t(M.nb) * BN;
  const double* src[NCH + 3];
#pragma unroll
  for (int c = 0; c < NCH; ++c) src[c] = c == 0 ? phi : pold;
#pragma unroll
  for (int c = 0; c < 3; ++c) src[NCH + c] = vel + c * n;
  auto getPhi = [&](int, int blk, int cell) { return phi[size_t(blk) * BN + cell]; };
  auto getPold = [&](int, int blk, int cell) { return pold[size_t(blk) * BN + cell]; };
  staged_blocks<NCH, 3>(M, src, nullptr, stage_smem, M.kerr, [&](int, int b, const StageMeta& m, double* st) {
    double* flab = st;
    double* olab = st + LG::V;
    const double* vin = st + NCH * LG::V;
    const double avg = M.case_sums ? M.case_sums[2 * M.bcase[b]] / M.case_sums[2 * M.bcase[b] + 1]
                                   : (sums ? sums[0] / sums[1] : 0.0);
    // the pressure of any cell of the mesh (coarse-fine flux correction)
    auto getP = [&](int, int blk, int cell) {
      const size_t i = size_t(blk) * BN + cell;
      const double p = phi[i] - avg;
      return USE_POLD ? p + pold[i] : p;
    };
    stage_fixup<1>(flab, M, m, getPhi, false);
    if (USE_POLD) stage_fixup<1>(olab, M, m, getPold, false);
    const bool fix = meta_has_finer(m);
    if (fix)
      for (int i = threadIdx.x; i < 3 * BN; i += NT) corr[i] = 0.0;
    __syncthreads();
    const double dtb = block_dt(M, b, dt);
    const double h = m.h, fac = -0.5 * dtb * h * h;
    auto P = [&](int x, int y, int z) {
      const int i = LG::at(x, y, z);
      const double p = flab[i] - avg;
      return USE_POLD ? p + olab[i] : p;
    };
    if (fix) {
      for (int f = 0; f < 6; ++f) {
        if (m.kind[f] != K_FINER) continue;
        const int d = f >> 1, s = f & 1;
        if (threadIdx.x < 64) {
          const int a = threadIdx.x & 7, bb = threadIdx.x >> 3;
          int q[3], g[3];
          face_lab_pair(d, s, a, bb, q, g);
          const int ch = m.nbr[4 * f + (a >> 2) + 2 * (bb >> 2)];
          const double hf = M.h[ch], facf = -0.5 * dtb * hf * hf;
          const double sg = s ? -1.0 : 1.0, sgc = -sg;
          double v = sg * fac * (P(g[0], g[1], g[2]) + P(q[0], q[1], q[2]));
#pragma unroll
          for (int e2 = 0; e2 < 2; ++e2)
#pragma unroll
            for (int e1 = 0; e1 < 2; ++e1) {
              const int fa = 2 * (a & 3) + e1, fb = 2 * (bb & 3) + e2;
              const int cf = face_cell(d, 1 - s, 0, fa, fb);
              const double pf = getP(0, ch, cf);
              const double gp = child_ghost1([&](int cell) { return getP(0, b, cell); }, M, ch, d, s, fa, fb);
              v += sgc * facf * (gp + pf);
            }
          corr[d * BN + face_cell(d, s, 0, a, bb)] += v;
        }
        __syncthreads();
      }
    }
    const double ih3 = 1.0 / (h * h * h);
    for (int qq = 0; qq < 2; ++qq) {
      const int cell = threadIdx.x + qq * NT;
      const int x = cell & 7, y = (cell >> 3) & 7, z = cell >> 6;
      const size_t gi = size_t(b) * BN + cell;
      double g0 = fac * (P(x + 1, y, z) - P(x - 1, y, z));
      double g1 = fac * (P(x, y + 1, z) - P(x, y - 1, z));
      double g2 = fac * (P(x, y, z + 1) - P(x, y, z - 1));
      if (fix) {
        g0 += corr[cell];
        g1 += corr[BN + cell];
        g2 += corr[2 * BN + cell];
      }
      vel[gi] = vin[cell] + ih3 * g0;
      vel[n + gi] = vin[BN + cell] + ih3 * g1;
      vel[2 * n + gi] = vin[2 * BN + cell] + ih3 * g2;
      pnew[gi] = P(x, y, z);
    }
    __syncthreads();
  });
}

template <int USE_POLD>
constexpr size_t grad_smem() {
  return StagedShape<1 + USE_POLD, 3>::kBytes + 3 * BN * sizeof(double);
}

int launch_grad_update(const DevMesh& M, double* vel, const double* phi, const double* pold, double* pnew,
                       const double* sums, double dt, int step, int step_2nd_start, int grid, cudaStream_t s) {
  static unsigned long long attr[2] = {0, 0};
  static int resident[2][64];
  int dev = 0;
  CUP_CUDA_TRY(cudaGetDevice(&dev));
  ProfScope ps("grad_update", s);
  if (step > step_2nd_start) {
    if (int rc = resident_ctas(k_grad_update<1>, grad_smem<1>(), attr[1], resident[1])) return rc;
    grid = std::max(1, std::min({grid, resident[1][dev], M.nb}));
    k_grad_update<1><<<grid, NT, grad_smem<1>(), s>>>(M, vel, phi, pold, pnew, sums, dt);
  } else {
    if (int rc = resident_ctas(k_grad_update<0>, grad_smem<0>(), attr[0], resident[0])) return rc;
    grid = std::max(1, std::min({grid, resident[0][dev], M.nb}));
    k_grad_update<0><<<grid, NT, grad_smem<0>(), s>>>(M, vel, phi, pold, pnew, sums, dt);
  }
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

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
