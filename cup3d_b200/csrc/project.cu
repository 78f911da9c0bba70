// The projection's two stencil passes on the device (FP64): the Poisson
// right-hand side and the gradient update.
//
// Both are bound by memory latency: 48 and 72 bytes a cell and a few dozen
// operations.  A warp takes half a block, four rows of eight z-columns; a
// thread keeps its column in registers and reads the x and y neighbours by
// plain loads, which hit L1 (the half block's own rows, or a neighbour's face
// row through a pointer chosen once per block).  No shared-memory tile and no
// barrier wider than the warp: every load of a block is independent of the
// others, and up to 32 warps of an SM overlap.  Only the ghosts that the
// stencils use are formed (one velocity component a face).  At coarse-fine
// faces the 32 or 64 face cells of the half block are spread over the lanes,
// which leave the ghosts (and at finer faces the flux corrections) in the
// warp's scratch for the lanes at the face.
#include <algorithm>

#include "../../include/cup3d_b200.h"
#include "lab.cuh"
#include "profiler.h"
#include "stencils.cuh"

namespace cup3d {

namespace {

constexpr int PT = 128;        // threads of a CTA: two blocks, a warp per half
constexpr int PBLOCKS = PT / 64;

// A warp's half block: rows gy = 4 half .. 4 half + 3.
struct Half {
  int b, half, lane, gx, gy;
  size_t own;     // the block's first cell
  int cell0;      // the thread's column
  int kinds;      // face kinds, 4 bits a face
  int nbr;        // lane i < 24: face-neighbour entry i
  int par;        // index parities, bit e for axis e
  __device__ __forceinline__ void load(const DevMesh& M, int block, int warp) {
    b = block;
    half = warp & 1;
    lane = threadIdx.x & 31;
    gx = lane & 7;
    gy = 4 * half + (lane >> 3);
    own = size_t(b) * BN;
    cell0 = gy * 8 + gx;
    int k = lane < 6 ? M.fkind[6 * b + lane] << (4 * lane) : 0;
    nbr = lane < 24 ? M.fnbr[24 * b + lane] : 0;
    const int i = lane < 3 ? M.index[3 * b + lane] & 1 : 0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) k |= __shfl_xor_sync(0xffffffffu, k, o);
    kinds = __shfl_sync(0xffffffffu, k, 0);
    par = int(__ballot_sync(0xffffffffu, i));
  }
  __device__ __forceinline__ int kind(int f) const { return (kinds >> (4 * f)) & 15; }
  __device__ __forceinline__ int nb(int f, int q = 0) const { return __shfl_sync(0xffffffffu, nbr, 4 * f + q); }
  // the neighbour at face cell (a, bb) (called by the whole warp)
  __device__ __forceinline__ int nb_at(int f, int a, int bb) const {
    return nb(f, kind(f) == K_FINER ? (a >> 2) + 2 * (bb >> 2) : 0);
  }
};

// Value of a neighbour of a column: at ptr + z * stride, times sign.
struct Edge {
  const double* ptr;
  int stride;
  double sign;
  __device__ __forceinline__ double at(int z) const { return sign * ptr[z * stride]; }
};

// A field read by block and cell: a - avg, plus b where given.
struct Field {
  const double* a;
  const double* b;
  double avg;
  __device__ __forceinline__ double operator()(int blk, int cell) const {
    const size_t i = size_t(blk) * BN + cell;
    const double v = a[i] - avg;
    return b ? v + b[i] : v;
  }
};

// Ghost at layer 1 beyond face f with a coarser or finer neighbour nb (the
// child at the cell, for a finer one), at face cell (a, bb): the lab rules of
// lab.cuh.  par: the block's index parities.  Out of line, as fine_sums: the
// coarse-fine faces' loads would take the registers of every block's path.
template <class V>
__device__ __noinline__ double cf_ghost(V F, int nb, int par, int kind, int f, int a, int bb) {
  const int d = f >> 1, s = f & 1;
  if (kind == K_FINER) {
    double sum = 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e)
      sum += F(nb, face_cell(d, 1 - s, e & 1, 2 * (a & 3) + ((e >> 1) & 1), 2 * (bb & 3) + (e >> 2)));
    return 0.125 * sum;
  }
  const int h1 = (par >> tan1(d)) & 1, h2 = (par >> tan2(d)) & 1;
  return c2f_ghost([&](int cell) { return F(nb, cell); }, d, s, 1, a, bb, h1, h2);
}

// Over the four fine cells at face cell (a, bb) of block b's finer face f
// (child ch): the sum of their values and the sum of their ghosts, which come
// from this block's own cells (child_ghost1); the four ghosts share their
// nodes, so their weights add up before the nodes are read.
__device__ __noinline__ double2 fine_sums(Field F, int b, int ch, int f, int a, int bb) {
  const int d = f >> 1, s = f & 1;
  double fine = 0.0, ghost = 0.0;
#pragma unroll
  for (int e = 0; e < 4; ++e) fine += F(ch, face_cell(d, 1 - s, 0, 2 * (a & 3) + (e & 1), 2 * (bb & 3) + (e >> 1)));
  int n1, n2;
  double wn[3], w1[3], w2[3];
  lagrange3(-0.25, wn);
  tan_sum(a, n1, w1);
  tan_sum(bb, n2, w2);
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 3; ++k) v = fma(wn[k], F(b, face_cell(d, s, k, n1 + i, n2 + j)), v);
      ghost = fma(w2[j] * w1[i], v, ghost);
    }
  return make_double2(fine, ghost);
}

// Scratch of a warp: per field the ghosts of the x faces (2 x 32, [row][z]),
// of the half's y face (64, [z][x]) and of the z faces (2 x 32, by lane); then
// the corrections likewise.
constexpr int kGhosts = 192;

// Runs body(face, kind, a, bb, slot) for the face cells of the half block on
// its coarse-fine faces, a cell a lane a turn.
template <class F>
__device__ __forceinline__ void cf_cells(const Half& H, F body) {
#pragma unroll 1
  for (int t = 0; t < 6; ++t) {
    // x faces, the half's y face in two turns, z faces
    const int f = t < 2 ? t : (t < 4 ? 2 + H.half : t);
    const int kind = H.kind(f);
    if (kind != K_COARSER && kind != K_FINER) continue;
    const int i = t == 3 ? H.lane + 32 : H.lane;
    const int a = t < 2 ? 4 * H.half + (i >> 3) : (t < 4 ? i & 7 : H.gx);
    const int bb = t < 2 ? i & 7 : (t < 4 ? i >> 3 : H.gy);
    body(f, kind, a, bb, t < 2 ? 32 * f + i : (t < 4 ? 64 + i : 32 * f + i));
  }
}

// The lower and upper x neighbours and the y neighbours of the thread's column
// of one field; g: the field's coarse-fine ghosts (null: taken as zero).  sgn:
// -1 where a boundary ghost changes sign (the normal velocity component).
__device__ __forceinline__ Edge edge_of(const Half& H, const double* v, const double* g, int f, double sgn) {
  const int d = f >> 1, s = f & 1;
  const int kind = H.kind(f), n = H.nb(f);
  const int step = d == 0 ? 1 : 8, pos = d == 0 ? H.gx : H.gy;
  Edge e{v + H.own + H.cell0 + (s ? step : -step), 64, 1.0};
  if (pos == (s ? BS - 1 : 0)) {
    if (kind == K_SAME) {
      e.ptr = v + size_t(n) * BN + H.cell0 + (s ? -7 * step : 7 * step);
    } else if (kind == K_BOUNDARY) {
      e.ptr = v + H.own + H.cell0;
      e.sign = sgn;
    } else if (!g) {
      e.sign = 0.0;
      e.ptr = v + H.own + H.cell0;
    } else if (d == 0) {
      e.ptr = g + 32 * s + 8 * (H.gy & 3);
      e.stride = 1;
    } else {
      e.ptr = g + 64 + H.gx;
      e.stride = 8;
    }
  }
  return e;
}

// The z neighbour beyond face f (4 or 5) of the thread's column.
__device__ __forceinline__ double z_end(const Half& H, const double* v, const double* g, int f, double sgn) {
  const int kind = H.kind(f), n = H.nb(f);
  if (kind == K_SAME) return v[size_t(n) * BN + H.cell0 + (f == 4 ? 7 * 64 : 0)];
  if (kind == K_BOUNDARY) return sgn * v[H.own + H.cell0 + (f == 4 ? 0 : 7 * 64)];
  return g ? g[32 * f + H.lane] : 0.0;
}

// u_def of one block, one component: the value of the body in slot sl where
// the grid's chi is its own (sl < 0: the block holds none).
struct Udef {
  const double* u;
  const double* body;
  const double* grid;
  __device__ __forceinline__ Udef(const ObstacleView& ob, const double* chi, int c, int blk, int sl)
      : u(sl < 0 ? nullptr : ob.udef + (size_t(c) * ob.nslots + sl) * BN),
        body(ob.chi + size_t(sl < 0 ? 0 : sl) * BN),
        grid(chi + size_t(blk) * BN) {}
  __device__ __forceinline__ double operator()(int, int cell) const {
    const double g = grid[cell], o = body[cell], v = u[cell];  // together: v does not wait for the test
    return g <= o ? v : 0.0;
  }
  __device__ __forceinline__ double at(int cell) const { return u ? (*this)(0, cell) : 0.0; }
  // the column of eight cells from `cell` on
  __device__ __forceinline__ void column(int cell, double (&v)[8]) const {
#pragma unroll
    for (int z = 0; z < 8; ++z) v[z] = 0.0;
    if (u)
#pragma unroll
      for (int z = 0; z < 8; ++z) v[z] = (*this)(0, cell + z * 64);
  }
};

// The divergence of u_def (differences of the two neighbours, not scaled) on
// the thread's column, to dv[8][32].  Component by component: a column comes
// with eight independent loads a field, the x and y neighbours from the lanes
// that hold them, and only the lanes at the half block's sides read on; gd: the
// coarse-fine ghosts.  (A neighbour at a time, 48 dependent calls a thread,
// the right-hand side next to a deforming body took 57 us on a box of 512
// blocks and 300 us on a refined mesh of 2624 blocks, 1519 of them with body
// cells; now 21 and 122, of which 12 and 64 without the deformation.)
__device__ __forceinline__ void udef_divergence(const Half& H, const ObstacleView& ob, const double* chi,
                                                const double* gd, double* dv) {
  const int sl = ob.slot[H.b];
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    double d[8], t[8];
    Udef(ob, chi, c, H.b, sl).column(H.cell0, d);
#pragma unroll
    for (int z = 0; z < 8; ++z) t[z] = c == 2 && z < 7 ? d[z + 1] : 0.0;
#pragma unroll
    for (int z = 1; z < 8; ++z) t[z] -= c == 2 ? d[z - 1] : 0.0;
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      const int f = 2 * c + s, kind = H.kind(f), n = H.nb(f);
      const double sg = s ? 1.0 : -1.0;
      if (c == 2) {
        double e;
        if (kind == K_SAME)
          e = Udef(ob, chi, c, n, ob.slot[n]).at(H.cell0 + (s ? 0 : 7 * 64));
        else if (kind == K_BOUNDARY)
          e = s ? -d[7] : -d[0];
        else
          e = gd[32 * f + H.lane];
        t[0] += s ? 0.0 : sg * e;
        t[7] += s ? sg * e : 0.0;
        continue;
      }
      const int step = c ? 8 : 1, row = H.lane >> 3;
      double w[8];
#pragma unroll
      for (int z = 0; z < 8; ++z) w[z] = __shfl_sync(0xffffffffu, d[z], H.lane + (s ? step : -step));
      const bool face = (c ? H.gy : H.gx) == (s ? BS - 1 : 0);  // at the block's face
      if (face || (c && row == (s ? 3 : 0))) {
        if (!face || kind == K_SAME) {
          const int blk = face ? n : H.b;
          Udef(ob, chi, c, blk, ob.slot[blk]).column(H.cell0 + (face ? (s ? -7 : 7) : (s ? 1 : -1)) * step, w);
        } else {
#pragma unroll
          for (int z = 0; z < 8; ++z)
            w[z] = kind == K_BOUNDARY ? -d[z] : gd[c ? 64 + H.gx + 8 * z : 32 * s + 8 * row + z];
        }
      }
#pragma unroll
      for (int z = 0; z < 8; ++z) t[z] += sg * w[z];
    }
#pragma unroll
    for (int z = 0; z < 8; ++z) dv[32 * z + H.lane] = c ? dv[32 * z + H.lane] + t[z] : t[z];
  }
}

// The u_def part of the flux correction at face cell (a, bb) of finer face f
// of a block next to a deforming body: chi times the face values, coarse and
// fine (kernelUpdateTmpV with the flux correction).  ch: the child there, gd:
// the block's ghost.  The four fine ghosts come from this block's cells and
// share their nodes (child_ghost1).
__device__ __noinline__ double udef_correction(ObstacleView ob, const double* chi, int b, int ch, int f, int a, int bb,
                                               double gd, double fac, double facf) {
  const int d = f >> 1, s = f & 1, oc = face_cell(d, s, 0, a, bb);
  const double sg = s ? -1.0 : 1.0;
  const Udef own(ob, chi, d, b, ob.slot[b]), fine(ob, chi, d, ch, ob.slot[ch]);
  double v = -sg * chi[size_t(b) * BN + oc] * fac * (gd + own.at(oc));
  int n1, n2;
  double wn[3], w1[2][3], w2[2][3], g[4] = {0.0, 0.0, 0.0, 0.0};
  lagrange3(-0.25, wn);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    tan_stencil(2 * (a & 3) + e, a >> 2, n1, w1[e]);
    tan_stencil(2 * (bb & 3) + e, bb >> 2, n2, w2[e]);
  }
  if (own.u)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        double q = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) q = fma(wn[k], own(b, face_cell(d, s, k, n1 + i, n2 + j)), q);
#pragma unroll
        for (int e = 0; e < 4; ++e) g[e] = fma(w2[e >> 1][j] * w1[e & 1][i], q, g[e]);
      }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int cf = face_cell(d, 1 - s, 0, 2 * (a & 3) + (e & 1), 2 * (bb & 3) + (e >> 1));
    v += sg * chi[size_t(ch) * BN + cf] * facf * (g[e] + fine.at(cf));
  }
  return v;
}

}  // namespace

// ---------------------------------------------------------------------------
// PressureProjection RHS: KernelPressureRHS (PressureProjection.cpp:96-199),
// kernelUpdateTmpV (:202-242) and KernelDivPressure (:16-94, step > 2).
// NEAR: blocks marked in ob.near subtract chi div u_def.
// ---------------------------------------------------------------------------
template <int USE_POLD, int NEAR>
__global__ void __launch_bounds__(PT, 6)
    k_pressure_rhs(DevMesh M, const double* __restrict__ vel, const double* __restrict__ pold,
                   const double* __restrict__ chi, ObstacleView ob, double dt, double* __restrict__ lhs,
                   double* __restrict__ phi) {
  // near a deforming body also u_def's ghosts and its divergence
  __shared__ double scratch[PT / 32][3 * kGhosts + (NEAR ? kGhosts + 8 * 32 : 0)];
  const int warp = threadIdx.x >> 5;
  double* gu = scratch[warp];
  double* gp = gu + kGhosts;
  double* corr = gp + kGhosts;
  double* gd = corr + kGhosts;
  double* dv = gd + kGhosts;
  const size_t n = size_t(M.nb) * BN;
  Half H;
  for (int b = blockIdx.x * PBLOCKS + (warp >> 1); b < M.nb; b += gridDim.x * PBLOCKS) {
    H.load(M, b, warp);
    const double h = M.h[b], dtb = block_dt(M, b, dt);
    const double fac = 0.5 * h * h / dtb;
    const bool near = NEAR && ob.near[b] != 0;
    auto U = [&](int d) { return Field{vel + d * n, nullptr, 0.0}; };
    const Field P{pold, nullptr, 0.0};
    // the correction of the right-hand side at a finer face's cell; gn, gq,
    // gs: the ghosts there of the velocity, p_old and u_def
    auto correction = [&](int f, int a, int bb, double gn, double gq, double gs) {
      const int d = f >> 1, s = f & 1, oc = face_cell(d, s, 0, a, bb), ch = H.nb_at(f, a, bb);
      const double hf = 0.5 * h, facf = 0.25 * fac;  // h = h0 2^-level: exact
      const double sg = s ? -1.0 : 1.0;
      const double2 u = fine_sums(U(d), b, ch, f, a, bb);
      double v = sg * fac * (gn + vel[d * n + H.own + oc]) - sg * facf * (u.y + u.x);
      if (USE_POLD) {
        const double2 p = fine_sums(P, b, ch, f, a, bb);
        v -= h * (pold[H.own + oc] - gq) + hf * (p.x - p.y);
      }
      if (near) v += udef_correction(ob, chi, b, ch, f, a, bb, gs, fac, facf);
      return v;
    };
    __syncwarp();  // the last block's lanes are done with the scratch
    cf_cells(H, [&](int f, int kind, int a, int bb, int i) {
      const int nb = H.nb_at(f, a, bb);
      const double u = cf_ghost(U(f >> 1), nb, H.par, kind, f, a, bb);
      const double p = USE_POLD ? cf_ghost(P, nb, H.par, kind, f, a, bb) : 0.0;
      double ud = 0.0;
      if (near) {
        const int sl = ob.slot[nb];
        if (sl >= 0) ud = cf_ghost(Udef(ob, chi, f >> 1, nb, sl), nb, H.par, kind, f, a, bb);
        gd[i] = ud;
      }
      gu[i] = u;
      if (USE_POLD) gp[i] = p;
      if (kind == K_FINER) corr[i] = correction(f, a, bb, u, p, ud);
    });
    __syncwarp();
    if (near) udef_divergence(H, ob, chi, gd, dv);
    const int fy = 2 + H.half;
    const double* w = vel + 2 * n + H.own + H.cell0;
    const Edge um = edge_of(H, vel, gu, 0, -1.0), up = edge_of(H, vel, gu, 1, -1.0);
    const Edge vm = edge_of(H, vel + n, gu, 2, -1.0), vp = edge_of(H, vel + n, gu, 3, -1.0);
    double wc[8], out[8];
#pragma unroll
    for (int z = 0; z < 8; ++z) wc[z] = w[z * 64];
    const double wm = z_end(H, vel + 2 * n, gu, 4, -1.0), wp = z_end(H, vel + 2 * n, gu, 5, -1.0);
#pragma unroll
    for (int z = 0; z < 8; ++z) {
      const double lo = z > 0 ? wc[z - 1] : wm, hi = z < 7 ? wc[z + 1] : wp;
      out[z] = fac * (up.at(z) - um.at(z) + vp.at(z) - vm.at(z) + hi - lo);
    }
    if (near)
#pragma unroll
      for (int z = 0; z < 8; ++z) out[z] += -chi[H.own + H.cell0 + z * 64] * fac * dv[32 * z + H.lane];
    if (USE_POLD) {
      double pc[8];
#pragma unroll
      for (int z = 0; z < 8; ++z) pc[z] = pold[H.own + H.cell0 + z * 64];
      const double pm = z_end(H, pold, gp, 4, 1.0), pp = z_end(H, pold, gp, 5, 1.0);
      const Edge xm = edge_of(H, pold, gp, 0, 1.0), xp = edge_of(H, pold, gp, 1, 1.0);
      const Edge ym = edge_of(H, pold, gp, 2, 1.0), yp = edge_of(H, pold, gp, 3, 1.0);
#pragma unroll
      for (int z = 0; z < 8; ++z) {
        const double lo = z > 0 ? pc[z - 1] : pm, hi = z < 7 ? pc[z + 1] : pp;
        out[z] -= h * (xp.at(z) + xm.at(z) + yp.at(z) + ym.at(z) + hi + lo - 6.0 * pc[z]);
      }
    }
    // the owners add the corrections, in face order
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (H.kind(s) == K_FINER && H.gx == (s ? 7 : 0))
#pragma unroll
        for (int z = 0; z < 8; ++z) out[z] += corr[32 * s + 8 * (H.gy & 3) + z];
    if (H.kind(fy) == K_FINER && H.gy == (H.half ? 7 : 0))
#pragma unroll
      for (int z = 0; z < 8; ++z) out[z] += corr[64 + H.gx + 8 * z];
    if (H.kind(4) == K_FINER) out[0] += corr[128 + H.lane];
    if (H.kind(5) == K_FINER) out[7] += corr[160 + H.lane];
    const size_t o = H.own + H.cell0;
#pragma unroll
    for (int z = 0; z < 8; ++z) {
      lhs[o + z * 64] = out[z];
      phi[o + z * 64] = 0.0;
    }
  }
}

static int project_grid(const DevMesh& M, int grid) {
  return std::max(1, std::min(grid, (M.nb + PBLOCKS - 1) / PBLOCKS));
}

int launch_pressure_rhs(const DevMesh& M, const double* vel, const double* pold, const double* chi,
                        const ObstacleView& ob, double dt, int step, int step_2nd_start, double* lhs, double* phi,
                        int grid, cudaStream_t s) {
  ProfScope ps("pressure_rhs", s);
  // with udef = 0 in every slot (rigid bodies) the near-body terms, chi times
  // the divergence of udef with its flux correction, are exact zeros
  const bool near = ob.near && ob.nslots > 0 && !ob.udef_zero;
  const int g = project_grid(M, grid);
  if (step > step_2nd_start) {
    if (near)
      k_pressure_rhs<1, 1><<<g, PT, 0, s>>>(M, vel, pold, chi, ob, dt, lhs, phi);
    else
      k_pressure_rhs<1, 0><<<g, PT, 0, s>>>(M, vel, pold, chi, ob, dt, lhs, phi);
  } else {
    if (near)
      k_pressure_rhs<0, 1><<<g, PT, 0, s>>>(M, vel, pold, chi, ob, dt, lhs, phi);
    else
      k_pressure_rhs<0, 0><<<g, PT, 0, s>>>(M, vel, pold, chi, ob, dt, lhs, phi);
  }
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// Mean removal + incremental pressure (PressureProjection.cpp:404-446) fused
// with KernelGradP (:244-323) and the velocity update (:451-467).  The
// pressure p = phi - avg (+ p_old) is formed at the point of use.
// ---------------------------------------------------------------------------
template <int USE_POLD>
__global__ void __launch_bounds__(PT, 6)
    k_grad_update(DevMesh M, double* __restrict__ vel, const double* __restrict__ phi, const double* __restrict__ pold,
                  double* __restrict__ pnew, const double* sums, double dt) {
  __shared__ double scratch[PT / 32][2 * kGhosts];
  const int warp = threadIdx.x >> 5;
  double* gp = scratch[warp];  // ghosts of phi + p_old
  double* corr = gp + kGhosts;
  const size_t n = size_t(M.nb) * BN;
  Half H;
  for (int b = blockIdx.x * PBLOCKS + (warp >> 1); b < M.nb; b += gridDim.x * PBLOCKS) {
    H.load(M, b, warp);
    const double h = M.h[b], dtb = block_dt(M, b, dt);
    const double avg = M.case_sums ? M.case_sums[2 * M.bcase[b]] / M.case_sums[2 * M.bcase[b] + 1]
                                   : (sums ? sums[0] / sums[1] : 0.0);
    const double fac = -0.5 * dtb * h * h;
    const Field Q{phi, USE_POLD ? pold : nullptr, 0.0}, P{phi, USE_POLD ? pold : nullptr, avg};
    auto correction = [&](int f, int a, int bb, double ghost) {
      const int d = f >> 1, s = f & 1;
      const double facf = 0.25 * fac;  // hf = h / 2
      const double2 p = fine_sums(P, b, H.nb_at(f, a, bb), f, a, bb);
      const double v = fac * (ghost + P(b, face_cell(d, s, 0, a, bb))) - facf * (p.y + p.x);
      return s ? -v : v;
    };
    __syncwarp();
    cf_cells(H, [&](int f, int kind, int a, int bb, int i) {
      const double q = cf_ghost(Q, H.nb_at(f, a, bb), H.par, kind, f, a, bb);
      gp[i] = q;
      if (kind == K_FINER) corr[i] = correction(f, a, bb, q - avg);
    });
    __syncwarp();
    const double ih3 = 1.0 / (h * h * h);
    const size_t o = H.own + H.cell0;
    double* u = vel + o;
    double pc[8];
#pragma unroll
    for (int z = 0; z < 8; ++z) {
      pc[z] = phi[o + z * 64] - avg;
      if (USE_POLD) pc[z] += pold[o + z * 64];
      pnew[o + z * 64] = pc[z];
    }
    {  // z
      double lo = z_end(H, phi, gp, 4, 1.0) - avg, hi = z_end(H, phi, gp, 5, 1.0) - avg;
      if (USE_POLD) {
        lo += z_end(H, pold, nullptr, 4, 1.0);
        hi += z_end(H, pold, nullptr, 5, 1.0);
      }
#pragma unroll
      for (int z = 0; z < 8; ++z) {
        double g = fac * ((z < 7 ? pc[z + 1] : hi) - (z > 0 ? pc[z - 1] : lo));
        if (z == 0 && H.kind(4) == K_FINER) g += corr[128 + H.lane];
        if (z == 7 && H.kind(5) == K_FINER) g += corr[160 + H.lane];
        u[2 * n + z * 64] += ih3 * g;
      }
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const Edge fm = edge_of(H, phi, gp, 2 * d, 1.0), fp = edge_of(H, phi, gp, 2 * d + 1, 1.0);
      double g[8];
      if (USE_POLD) {
        // the scratch holds phi + p_old: nothing to add at its lanes
        const Edge om = edge_of(H, pold, nullptr, 2 * d, 1.0), op = edge_of(H, pold, nullptr, 2 * d + 1, 1.0);
#pragma unroll
        for (int z = 0; z < 8; ++z) g[z] = ((fp.at(z) - avg) + op.at(z)) - ((fm.at(z) - avg) + om.at(z));
      } else {
#pragma unroll
        for (int z = 0; z < 8; ++z) g[z] = (fp.at(z) - avg) - (fm.at(z) - avg);
      }
#pragma unroll
      for (int z = 0; z < 8; ++z) g[z] *= fac;
      if (d == 0) {
#pragma unroll
        for (int s = 0; s < 2; ++s)
          if (H.kind(s) == K_FINER && H.gx == (s ? 7 : 0))
#pragma unroll
            for (int z = 0; z < 8; ++z) g[z] += corr[32 * s + 8 * (H.gy & 3) + z];
      } else if (H.kind(2 + H.half) == K_FINER && H.gy == (H.half ? 7 : 0)) {
#pragma unroll
        for (int z = 0; z < 8; ++z) g[z] += corr[64 + H.gx + 8 * z];
      }
#pragma unroll
      for (int z = 0; z < 8; ++z) u[d * n + z * 64] += ih3 * g[z];
    }
  }
}

int launch_grad_update(const DevMesh& M, double* vel, const double* phi, const double* pold, double* pnew,
                       const double* sums, double dt, int step, int step_2nd_start, int grid, cudaStream_t s) {
  ProfScope ps("grad_update", s);
  const int g = project_grid(M, grid);
  if (step > step_2nd_start)
    k_grad_update<1><<<g, PT, 0, s>>>(M, vel, phi, pold, pnew, sums, dt);
  else
    k_grad_update<0><<<g, PT, 0, s>>>(M, vel, phi, pold, pnew, sums, dt);
  CUP_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace cup3d
