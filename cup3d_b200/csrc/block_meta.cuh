// A block's entries of the mesh tables staged in shared memory: the kernel
// that walks blocks asks for the next one's while it computes the present one,
// so that no copy of a block waits on a table load.
#pragma once
#include "async_copy.cuh"
#include "lab.cuh"

namespace cup3d {

// One block's table entries, staged by cp.async.
struct StageMeta {
  int kind[6];
  int nbr[24];
  int index[3];
  int pad_;
  double h;
};
static_assert(sizeof(StageMeta) == 144, "StageMeta layout");

// Issues the copies of block b's table entries into m (threads 0..33).
__device__ __forceinline__ void meta_issue(StageMeta* m, const DevMesh& M, int b) {
  const int t = threadIdx.x;
  if (t < 6)
    cp_async4(&m->kind[t], M.fkind + 6 * b + t);
  else if (t < 30)
    cp_async4(&m->nbr[t - 6], M.fnbr + 24 * b + (t - 6));
  else if (t < 33)
    cp_async4(&m->index[t - 30], M.index + 3 * b + (t - 30));
  else if (t == 33)
    cp_async8(&m->h, M.h + b);
}

// The same with plain loads (a CTA's first block).
__device__ __forceinline__ void meta_load(StageMeta* m, const DevMesh& M, int b) {
  const int t = threadIdx.x;
  if (t < 6)
    m->kind[t] = M.fkind[6 * b + t];
  else if (t < 30)
    m->nbr[t - 6] = M.fnbr[24 * b + (t - 6)];
  else if (t < 33)
    m->index[t - 30] = M.index[3 * b + (t - 30)];
  else if (t == 33)
    m->h = M.h[b];
}

}  // namespace cup3d
