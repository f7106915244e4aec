// Geometry and host interface of the resident solve (cg_res.cuh, cg_res.cu).
#ifndef FREHD_CG_RES_H
#define FREHD_CG_RES_H

#include <cuda_runtime.h>

#include "cg1.h"
#include "domain.cuh"

namespace frehd {

constexpr int kResTW = 64;              // tile width: a warp's 32 lanes, two cells each
constexpr int kResPitch = kResTW + 4;   // shared-memory row: the tile and two cells on each side
constexpr int kResMaxKR = 4;            // rows per thread: tiles 64 x 16, 64 x 32, 64 x 64
constexpr int kResSlot = 8;             // entries per CTA in the reduction buffer
constexpr int kResMaxOuter = 8;         // refinements of one mixed-precision solve

__host__ __device__ constexpr int res_th(int KR) { return 16 * KR; }
__host__ __device__ constexpr int res_edge(int KR) { return 2 * res_th(KR) + 2 * kResTW + 4; }
__host__ __device__ inline int res_ntx(int nx) { return (nx + kResTW - 1) / kResTW; }
__host__ __device__ inline long res_tiles(int nx, int ny, int KR) {
  return (long)res_ntx(nx) * ((ny + res_th(KR) - 1) / res_th(KR));
}
// Rows per thread of a solve on at most `ctas` CTAs: the smallest tile that
// covers the domain (the least work between two reductions); 0 if none does.
__host__ __device__ inline int res_rows(int nx, int ny, long ctas) {
  for (int KR = 1; KR <= kResMaxKR; KR *= 2)
    if (res_tiles(nx, ny, KR) <= ctas) return KR;
  return 0;
}
// 16-byte entries of a solve's exchange buffer (both parities): the CTAs' sums,
// then the tiles' outer rows and columns.
__host__ __device__ inline long res_entries(long ntiles, int KR) {
  return 2 * ntiles * (kResSlot + (long)res_edge(KR));
}
__host__ __device__ constexpr unsigned res_smem(int KR) {
  return 2u * (res_th(KR) + 4) * kResPitch * 8u;
}

// CTAs of the resident solve that fit on the device at once (also raises the
// kernels' shared-memory limits).
int cgr_capacity(int device, int *ctas);
// Exchange bytes of a domain's solve with `rows` rows per thread or more.
long long cgr_exchange_bytes(const Grid &g, int rows);
// The domain's solve on its own (rows from res_rows of the capacity).
int cgr_launch(const View &w, int rows, int x0_surface, int eliminate, cudaStream_t stream);
// Batched: CTA c runs jobs[job_start[c] .. job_start[c+1]) in order, then
// single-CTA jobs from `singles` (*taken zero at the launch).  Every CTA's list
// keeps the domains in one common order, so that no two groups wait for each
// other.  CgJob::flags bits 4 and up: rows per thread.
int cgr_launch_batch(const View *views2, const int *job_start, const CgJob *jobs, const CgJob *singles,
                     int nsingles, int *taken, int nctas, int any_mixed, cudaStream_t stream);

}  // namespace frehd

#endif
