// Geometry and host interface of the resident solve (cg_res.cuh, cg_res.cu).
#ifndef FREHD_CG_RES_H
#define FREHD_CG_RES_H

#include <cuda_runtime.h>

#include "cg1.h"
#include "domain.cuh"

namespace frehd {

constexpr int kResTW = 64;              // tile width: a warp's 32 lanes, two cells each
constexpr int kResPitch = kResTW + 4;   // shared-memory row: the tile and two cells on each side
constexpr int kResWarps = 16, kResThreads = 32 * kResWarps;
constexpr int kResMinKR = 1, kResMaxKR = 4;  // rows per thread: tiles 64 x 16, 64 x 32, 64 x 64
constexpr int kResSlot = 8;             // entries per CTA in the reduction buffer (six sums)
constexpr int kResFlat = 16;            // CTAs whose sums are added in one go, and the largest cluster
constexpr int kResMaxOuter = 8;         // refinements of one mixed-precision solve
// With more CTAs than kResFlat: how many form a group, and a cluster.  Eight, while they
// fit the device (clusters of eight leave 120 of the 148 SMs usable, of four 132).
constexpr int kResMaxGroups = 32, kResEights = 112, kResClustered = 4 * kResMaxGroups;
__host__ __device__ constexpr int res_group(int nb) { return nb <= kResEights ? 8 : 4; }
__host__ __device__ constexpr int res_th(int KR) { return kResWarps * KR; }
__host__ __device__ constexpr int res_edge(int KR) { return 2 * res_th(KR) + 2 * kResTW + 4; }
__host__ __device__ inline int res_ntx(int nx) { return (nx + kResTW - 1) / kResTW; }
__host__ __device__ inline long res_tiles(int nx, int ny, int KR) {
  return (long)res_ntx(nx) * ((ny + res_th(KR) - 1) / res_th(KR));
}
// Rows per thread of a solve on at most `ctas` CTAs: the smallest tile that
// covers the domain (the least work between two reductions); 0 if none does.
__host__ __device__ inline int res_rows(int nx, int ny, long ctas) {
  for (int KR = kResMinKR; KR <= kResMaxKR; KR *= 2)
    if (res_tiles(nx, ny, KR) <= ctas) return KR;
  return 0;
}
// 16-byte entries of a solve's exchange buffer (both parities): the CTAs' sums, the
// groups' sums, then the tiles' outer rows and columns.
__host__ __device__ inline long res_entries(long ntiles, int KR) {
  return 2 * (ntiles * (kResSlot + (long)res_edge(KR)) + kResSlot * kResMaxGroups);
}
constexpr int kResSums = 6;             // sums of one iteration
// Shared memory of a CTA: every thread's part of the sums, then three FP64 arrays of
// the tile and two cells around it (set-up: sqrt|Ct| and the couplings; the solve uses
// the first, or the first two as four FP32 arrays), then the entries that the other
// CTAs of its cluster write (res_inbox: sums, totals, edges of both parities).
__host__ __device__ constexpr int res_arr(int KR) { return (res_th(KR) + 4) * kResPitch; }
__host__ __device__ constexpr int res_inbox(int KR) { return 2 * (kResSlot * (kResFlat + 1) + res_edge(KR)); }
__host__ __device__ constexpr unsigned res_smem(int KR) {
  return 8u * (kResSums * kResThreads + 3u * res_arr(KR)) + 16u * res_inbox(KR);
}

// The system of one solve.  Cell (i, j) at off + j * pitch + i of every array; nothing
// outside 0 <= i < nx, 0 <= j < ny is read, but for a mixed solve, whose residual reads
// the ghost ring of a domain's padded layout (res_residual_padded).
struct ResSys {
  int nx, ny;
  long pitch, off;
  const double *Ct, *Gx, *Gy, *b, *x0;  // x0 null: the solve starts from zero
  double *x;
  double eps;
  int max_iter, eliminate;
  Scratch *sc;
  uint4 *xbuf;
  unsigned *beat;  // counts on while the solve proceeds (null: nobody looks)
};

// CTAs of the resident solve that fit on the device at once, and how many of them in
// clusters of res_group (at most kResClustered).  Also raises the kernels'
// shared-memory limits.
int cgr_capacity(int device, int *ctas, int *clustered);
// Exchange bytes of a domain's solve with `rows` rows per thread or more.
long long cgr_exchange_bytes(const Grid &g, int rows);
// The domain's solve on its own (rows from res_rows of the capacity).  plain: without the
// clusters that the kernel expects (frehd_domain_set_solve_test).
int cgr_launch(const View &w, int rows, int clustered, bool plain, int x0_surface, int eliminate,
               cudaStream_t stream);
// The same for a system in any layout, in FP64.  s.xbuf: res_entries of its tiles, no
// entry of which carries a tag above s.sc->res_tag.
int cgr_launch_sys(const ResSys &s, int rows, int clustered, cudaStream_t stream);
// Batched: CTA c runs jobs[job_start[c] .. job_start[c+1]) in order, then
// single-CTA jobs from `singles` (*taken zero at the launch).  Every CTA's list
// keeps the domains in one common order, so that no two groups wait for each
// other.  CgJob::flags bits 4 and up: rows per thread.  bsync: the batch's counters
// (taken zero at the launch, and every domain's Scratch::res_arrived).
int cgr_launch_batch(const View *views2, const int *job_start, const CgJob *jobs, const CgJob *singles,
                     int nsingles, Scratch *bsync, int nctas, int any_mixed, cudaStream_t stream);

}  // namespace frehd

#endif
