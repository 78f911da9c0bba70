// AdvectionDiffusion on the device: one RK3 stage fused with its update
// (KernelAdvectDiffuse, AdvectionDiffusion.cpp:19-215, and the low-storage
// update of AdvectionDiffusion.cpp:286-320), FP64.
//
// A CTA of 192 threads takes one 8^3 block at a time: 64 threads per velocity
// component, each the owner of one line of 8 cells in the direction being
// differenced (x, then y, then z).  A thread reads the 14 values of its line
// (8 cells and 3 ghosts on either side) from shared memory once, sweeps the
// line in registers and adds the direction's contribution to the block's
// accumulator in shared memory; the z sweep, whose lines are coalesced
// columns, writes the result.
//
// What bounds it: WENO5 the FP64 pipe and issue slots (43% and 58% busy; 90 us a
// stage on the 2340-block sphere mesh), upwind5 the L2 traffic of the block and
// its ghosts (39 KB in, 24 KB out a block).  The layout serves the sweeps: rows
// padded to 9 values and planes to 72, so that the lines of a half-warp fall
// into different banks in x and y; ghost layers apart, [face][layer][line],
// read by the line's own index in all three directions, so that one rolled loop
// runs them all (three unrolled copies overflow the instruction cache).  55 KB
// of shared memory and 80 registers let four CTAs stay on an SM, whose copies
// and sweeps overlap.
#include "../../include/cup3d_b200.h"
#include "profiler.h"
#include "block_meta.cuh"
#include "stencils.cuh"

namespace cup3d {

namespace {

constexpr int AT = 192;          // threads: 3 components x 64 lines
constexpr int ROW = 9;           // padded row and plane of the staged block
constexpr int PLANE = 72;
constexpr int CELLS = 8 * PLANE;  // one component's staged cells
constexpr int LAYER = 68;         // padded ghost layer of 64
constexpr int GFACE = 2 * LAYER + 64;  // one face's three layers
constexpr int GHOSTS = 6 * GFACE;

struct UInf {
  double v[3];
};

struct AdvectSmem {
  double in[3][CELLS];
  double gh[3][GHOSTS];  // [face][layer][line]
  double acc[3][CELLS];  // tmpV, then the sum over the directions
  StageMeta meta[2];
  double fac[4];  // the block's advection, diffusion, fine diffusion and update factors
};

__device__ __forceinline__ double sq(double a) { return a * a; }

// The lines of direction d: the offset of line (a, b) (tangential coordinates
// in increasing dimension order) and the stride along it.
__device__ __forceinline__ int line_base(int d, int a, int b) {
  return d == 0 ? b * PLANE + a * ROW : (d == 1 ? b * PLANE + a : b * ROW + a);
}
__device__ __forceinline__ int line_stride(int d) { return d == 0 ? 1 : (d == 1 ? ROW : PLANE); }

// Barrier of one component's 64 threads.
__device__ __forceinline__ void comp_sync(int c) { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + c), "r"(64) : "memory"); }

// WENO5 (weno5_plus / weno5_minus of AdvectionDiffusion.cpp:32-64) on one
// line.  With the differences d_m = v_m - v_(m-1), the smoothness indicator
// of the three cells around m depends only on the place the face takes in
// them (left, middle, right), not on the upwind side:
//   4 b = 13/3 (d_(m+1) - d_m)^2 + t^2,  t = 3 d_(m+1) - d_m  (face right of the three),
//   d_m + d_(m+1)  (in the middle),  d_(m+1) - 3 d_m  (face left of the three),
// so q = (4 b + 4 eps)^2 is formed once per cell and place and serves both
// sides and both faces.  A face's value is the upwind cell's plus
//   G = (q2 q3 g1 + q1 (6 q3 g2 + 3 q2 g3)) / (q2 q3 + q1 (6 q3 + 3 q2)),
// the weights d_k / q_k (d = 0.1, 0.6, 0.3) over one denominator and g_k the
// candidate stencils less the upwind cell, in the same differences.
//
// The window moves along the line one face at a time.  At the face between
// cells p and p + 1 it holds d_(p-1) .. d_(p+3) and, per side, the q of the
// three stencils: (left p-1, middle p, right p+1) from below and
// (right p+2, middle p+1, left p) from above.
struct Weno {
  double d0, d1, d2, d3, d4;  // d_(p-1) .. d_(p+3)
  double k0, k1, k2;          // 13/3 (d_(m+1) - d_m)^2 + 4 eps of m = p, p+1, p+2
  double ql0, ql1, qm0, qm1, qr0, qr1;  // left p-1, p; middle p, p+1; right p+1, p+2
  static __device__ __forceinline__ double curv(double a, double b) {
    const double s = b - a;
    return fma((13.0 / 3.0) * s, s, 4e-6);
  }
  static __device__ __forceinline__ double left(double a, double b, double k) {
    const double t = fma(3.0, b, -a);
    return sq(fma(t, t, k));
  }
  static __device__ __forceinline__ double mid(double a, double b, double k) {
    const double t = a + b;
    return sq(fma(t, t, k));
  }
  static __device__ __forceinline__ double right(double a, double b, double k) {
    const double t = fma(-3.0, a, b);
    return sq(fma(t, t, k));
  }
  // the window at the face between v2 and v3 of the line v0 .. v5
  __device__ __forceinline__ void start(double v0, double v1, double v2, double v3, double v4, double v5) {
    d0 = v1 - v0;
    d1 = v2 - v1;
    d2 = v3 - v2;
    d3 = v4 - v3;
    d4 = v5 - v4;
    k0 = curv(d1, d2);
    k1 = curv(d2, d3);
    k2 = curv(d3, d4);
    ql0 = left(d0, d1, curv(d0, d1));
    ql1 = left(d1, d2, k0);
    qm0 = mid(d1, d2, k0);
    qm1 = mid(d2, d3, k1);
    qr0 = right(d2, d3, k1);
    qr1 = right(d3, d4, k2);
  }
  // to the next face; dn: the line's next difference
  __device__ __forceinline__ void advance(double dn) {
    d0 = d1;
    d1 = d2;
    d2 = d3;
    d3 = d4;
    d4 = dn;
    k0 = k1;
    k1 = k2;
    k2 = curv(d3, d4);
    ql0 = ql1;
    ql1 = left(d1, d2, k0);
    qm0 = qm1;
    qm1 = mid(d2, d3, k1);
    qr0 = qr1;
    qr1 = right(d3, d4, k2);
  }
  // G at the face from the upwind side `pos`
  __device__ __forceinline__ double face(bool pos) const {
    const double q1 = pos ? ql0 : qr1, q2 = pos ? qm0 : qm1, q3 = pos ? qr0 : ql1;
    const double e1 = pos ? d0 : d4, e2 = pos ? d1 : d3, e4 = pos ? d3 : d1;
    const double g1 = fma(5.0 / 6.0, e2, (-1.0 / 3.0) * e1);
    const double g2 = fma(1.0 / 6.0, e2, (1.0 / 3.0) * d2);
    const double g3 = fma(2.0 / 3.0, d2, (-1.0 / 6.0) * e4);
    const double q23 = q2 * q3, w2 = 6.0 * q3, w3 = 3.0 * q2;
    const double num = fma(q1, fma(w3, g3, w2 * g2), q23 * g1);
    const double den = fma(q1, w2 + w3, q23);
    return num / den;
  }
};

}  // namespace

template <int SCHEME>
__global__ void __launch_bounds__(AT, 4)
    k_advect_stage(DevMesh M, const double* __restrict__ vin, double* __restrict__ vout, double* __restrict__ tmpV,
                   double dt, double nu, UInf ui, int stage) {
  extern __shared__ __align__(16) unsigned char advect_smem[];
  AdvectSmem& S = *reinterpret_cast<AdvectSmem*>(advect_smem);
  const int c = threadIdx.x >> 6, lane = threadIdx.x & 63;
  const int la = lane & 7, lb = lane >> 3;
  const size_t n = size_t(M.nb) * BN;
  const double* vc = vin + c * n;
  double* in = S.in[c];
  double* gh = S.gh[c];
  double* acc = S.acc[c];
  const double alpha = stage == 0 ? 1.0 / 3.0 : (stage == 1 ? 15.0 / 16.0 : 8.0 / 15.0);
  const double beta = stage == 0 ? -5.0 / 9.0 : (stage == 1 ? -153.0 / 128.0 : 0.0);
  int it = 0;
  if (int(blockIdx.x) < M.nb) meta_load(&S.meta[0], M, blockIdx.x);
  __syncthreads();
  for (int b = blockIdx.x; b < M.nb; b += gridDim.x, ++it) {
    const StageMeta& m = S.meta[it & 1];
    const size_t own = size_t(b) * BN;
    // ---- the block, tmpV and the same-level ghosts by asynchronous copies
#pragma unroll
    for (int k = 0; k < 8; ++k) cp_async8(&in[k * PLANE + lb * ROW + la], vc + own + k * 64 + lane);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double* a = &acc[k * PLANE + lb * ROW + la];
      if (stage)
        cp_async8(a, tmpV + c * n + own + k * 64 + lane);
      else
        *a = 0.0;
    }
    bool second = false;  // faces whose ghosts need the staged block or a coarse layer
#pragma unroll 1
    for (int f = 0; f < 6; ++f) {
      const int kind = m.kind[f], d = f >> 1, s = f & 1;
      double* g = gh + f * GFACE;
      if (kind == K_SAME) {
        // one warp a face: in x four lanes a row of the neighbour (its four
        // nearest cells are one 32-byte sector), in y and z 16 bytes a lane
        // (a lane per cell and layer touched each row's line three times:
        // twice the wavefronts)
        const double* src = vc + size_t(m.nbr[4 * f]) * BN;
        const int l32 = lane & 31;
        if ((lane >> 5) != s) continue;
        if (d == 0) {
          const int x = (l32 & 3) + (s ? 0 : 4), l = s ? x : 7 - x;
          if (l < 3)
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int row = (l32 >> 2) + 8 * k;
              cp_async8(g + l * LAYER + row, src + 8 * row + x);
            }
        } else {
          const int x = 2 * (l32 & 3), r = l32 >> 2;  // r: z of a y face, y of a z face
#pragma unroll
          for (int l = 0; l < 3; ++l) {
            const int at = s ? l : 7 - l;
            cp_async16(g + l * LAYER + 8 * r + x, src + (d == 1 ? 64 * r + 8 * at : 64 * at + 8 * r) + x);
          }
        }
      } else if (kind == K_FINER) {
        const double* src = vc + size_t(m.nbr[4 * f + (la >> 2) + 2 * (lb >> 2)]) * BN;
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          double sum = 0.0;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            sum += src[face_cell(d, 1 - s, 2 * l + (e & 1), 2 * (la & 3) + ((e >> 1) & 1), 2 * (lb & 3) + (e >> 2))];
          g[l * LAYER + lane] = 0.125 * sum;
        }
      } else if (kind == K_COARSER) {
        // the coarse neighbour's three layers at its face cell (la, lb),
        // combined along the normal for each ghost layer (lagrange3 at -1/4, 1/4, 3/4)
        const double* src = vc + size_t(m.nbr[4 * f]) * BN;
        const double v0 = src[face_cell(d, 1 - s, 0, la, lb)], v1 = src[face_cell(d, 1 - s, 1, la, lb)],
                     v2 = src[face_cell(d, 1 - s, 2, la, lb)];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          double w[3];
          lagrange3((l - 0.5) * 0.5, w);
          g[l * LAYER + lane] = w[0] * v0 + w[1] * v1 + w[2] * v2;
        }
        second = true;
      } else {
        second = true;
      }
    }
    if (b + int(gridDim.x) < M.nb) meta_issue(&S.meta[(it + 1) & 1], M, b + gridDim.x);
    cp_async_commit();
    if (threadIdx.x == 0) {  // one thread's divisions, not everybody's
      const double h = m.h, h3 = h * h * h, hf = 0.5 * h;  // h = h0 2^-level: exact
      const double dtb = block_dt(M, b, dt);
      S.fac[0] = -dtb / h * h3 / (SCHEME == 1 ? 1.0 : 60.0);  // upwind5's derivative carries its 1/60 here
      S.fac[1] = (nu / h) * (dtb / h) * h3;
      S.fac[2] = (nu / hf) * (dtb / hf) * hf * hf * hf;
      S.fac[3] = alpha / h3;
    }
    cp_async_wait<0>();
    __syncthreads();
    if (second) {  // the same for the whole CTA
#pragma unroll 1
      for (int f = 0; f < 6; ++f) {
        const int kind = m.kind[f], d = f >> 1, s = f & 1;
        double* g = gh + f * GFACE;
        if (kind == K_BOUNDARY) {
          double v = in[line_base(d, la, lb) + (s ? 7 : 0) * line_stride(d)];
          if (m.nbr[4 * f] == BCK_WALL || c == d) v = -v;
          g[lane] = g[LAYER + lane] = g[2 * LAYER + lane] = v;
        } else if (kind == K_COARSER) {
          int n1, n2;
          double w1[3], w2[3], out[3] = {0.0, 0.0, 0.0};
          tan_stencil(la, m.index[tan1(d)] & 1, n1, w1);
          tan_stencil(lb, m.index[tan2(d)] & 1, n2, w2);
#pragma unroll
          for (int l = 0; l < 3; ++l)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const double* r = g + l * LAYER + 8 * (n2 + j) + n1;
              out[l] = fma(w2[j], w1[0] * r[0] + w1[1] * r[1] + w1[2] * r[2], out[l]);
            }
          comp_sync(c);  // every thread has read the coarse layer
#pragma unroll
          for (int l = 0; l < 3; ++l) g[l * LAYER + lane] = out[l];
        }
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
      const int base = line_base(d, la, lb), st = line_stride(d);
      const double* glo = gh + 2 * d * GFACE + lane;
      // flux correction at finer faces: this block's own diffusive face value
      // plus the four fine ones, whose ghosts come from this block's cells
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        if (m.kind[2 * d + s] != K_FINER) continue;
        const int* nbr = m.nbr + 4 * (2 * d + s);
        const double* ch = vc + size_t(nbr[(la >> 2) + 2 * (lb >> 2)]) * BN;
        double uf = 0.0;
#pragma unroll
        for (int e = 0; e < 4; ++e) uf += ch[face_cell(d, 1 - s, 0, 2 * (la & 3) + (e & 1), 2 * (lb & 3) + (e >> 1))];
        int n1, n2;
        double wn[3], w1[3], w2[3], gf = 0.0;
        lagrange3(-0.25, wn);
        tan_sum(la, n1, w1);
        tan_sum(lb, n2, w2);
        const int first = s ? 7 * st : 0, step = s ? -st : st;
#pragma unroll 1
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const double* q = in + line_base(d, n1 + i, n2 + j) + first;
            gf = fma(w2[j] * w1[i], wn[0] * q[0] + wn[1] * q[step] + wn[2] * q[2 * step], gf);
          }
        acc[base + first] += S.fac[1] * (in[base + first] - glo[s * GFACE]) + S.fac[2] * (uf - gf);
      }
      // the line: three ghosts, the eight cells, three ghosts
      const double* line = in + base;
      auto value = [&](int k) {
        return k < 3 ? glo[(2 - k) * LAYER] : (k < 11 ? line[(k - 3) * st] : glo[GFACE + (k - 11) * LAYER]);
      };
      const double* ud = S.in[d] + base;
      const double facA = S.fac[0], facD = S.fac[1];
      const double ud0 = d == 0 ? ui.v[0] : (d == 1 ? ui.v[1] : ui.v[2]);
      double* al = acc + base;
      if (SCHEME == 1) {
        Weno W;
        double last = value(5);
        W.start(value(0), value(1), value(2), value(3), value(4), last);
        double U = ud[0] + ud0;
        bool pos = U > 0;
        double G = W.face(pos);  // the first cell's lower face
        unsigned flips = 0;      // cells whose upwind side is not that of the cell below
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double v = value(i + 6);
          const double below = W.d2;  // the cell's difference to the one below
          W.advance(v - last);
          last = v;
          const double up = W.face(pos);
          const double der = pos ? below + (up - G) : W.d2 - (up - G);
          al[i * st] += facA * (U * der) + facD * (W.d2 - below);
          if (i < 7) {
            U = ud[(i + 1) * st] + ud0;
            const bool next = U > 0;
            if (next != pos) flips |= 2u << i;
            G = next != pos ? 0.0 : up;
            pos = next;
          }
        }
        // the lower faces of the cells where the side flips, from the cell's
        // own side, a cell a turn: a lane has few, the lanes of a warp have
        // them at different cells
        while (flips) {
          const int i = __ffs(flips) - 1;
          flips &= flips - 1;
          W.start(value(i), value(i + 1), value(i + 2), value(i + 3), value(i + 4), value(i + 5));
          U = ud[i * st] + ud0;
          pos = U > 0;
          G = W.face(pos);
          al[i * st] += facA * (U * (pos ? -G : G));
        }
      } else {
        double um3 = value(0), um2 = value(1), um1 = value(2), u = value(3), up1 = value(4), up2 = value(5);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double up3 = value(i + 6);
          const double U = ud[i * st] + ud0;
          const bool pos = U > 0;
          const double m3 = pos ? um3 : up3, m2 = pos ? um2 : up2, m1 = pos ? um1 : up1;
          const double p1 = pos ? up1 : um1, p2 = pos ? up2 : um2;
          const double der = -2 * m3 + 15 * m2 - 60 * m1 + 20 * u + 30 * p1 - 3 * p2;
          al[i * st] += facA * ((pos ? U : -U) * der) + facD * ((up1 - u) - (u - um1));
          um3 = um2;
          um2 = um1;
          um1 = u;
          u = up1;
          up1 = up2;
          up2 = up3;
        }
      }
      if (d < 2) comp_sync(c);  // the component's lines of the next direction cross these
    }
    // the thread's z column, complete
    const double fac = S.fac[3];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int at = lb * ROW + la + i * PLANE;
      const size_t gi = c * n + own + i * 64 + lane;
      const double tot = acc[at];
      vout[gi] = in[at] + tot * fac;
      if (stage < 2) tmpV[gi] = tot * beta;
    }
    __syncthreads();  // the stage is free for the next block
  }
}

int launch_advect_stage(const DevMesh& M, const double* vin, double* vout, double* tmpV, double dt, double nu,
                        const double* uinf, int scheme, int stage, int grid, cudaStream_t s) {
  const size_t smem = sizeof(AdvectSmem);
  static unsigned long long attr_set[2] = {0, 0};
  UInf ui{{uinf[0], uinf[1], uinf[2]}};
  if (scheme == 1) {
    if (first_on_device(attr_set[1]))
      CUP_CUDA_TRY(cudaFuncSetAttribute(k_advect_stage<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    ProfScope ps("advect_stage_weno5", s);
    k_advect_stage<1><<<grid, AT, smem, s>>>(M, vin, vout, tmpV, dt, nu, ui, stage);
  } else {
    if (first_on_device(attr_set[0]))
      CUP_CUDA_TRY(cudaFuncSetAttribute(k_advect_stage<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    ProfScope ps("advect_stage_upwind5", s);
    k_advect_stage<0><<<grid, AT, smem, s>>>(M, vin, vout, tmpV, dt, nu, ui, stage);
  }
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace cup3d
