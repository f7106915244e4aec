// Kernels of the resident solve (cg_res.cuh): one domain, or many in a batch.
#include "cg_res.cuh"

#include "frehd_internal.h"

namespace frehd {

namespace {

__device__ __forceinline__ void sys_of(const View &w, int x0_surface, int eliminate, ResSys *s) {
  s->nx = w.gr.nx;
  s->ny = w.gr.ny;
  s->pitch = w.gr.pitch;
  s->off = w.gr.at(0, 0);
  s->Ct = w.Ct;
  s->Gx = w.Gx;
  s->Gy = w.Gy;
  s->b = w.b;
  s->x0 = x0_surface ? w.surf_cur : nullptr;
  s->x = w.x;
  s->eps = w.p.eps;
  s->max_iter = w.p.maxIter;
  s->eliminate = eliminate;
  s->sc = w.sc;
  s->xbuf = w.xch;
}

// The domain's solve in its configured precision by nb CTAs.
template <int KR, bool kMix>
__device__ __forceinline__ bool res_solve(const ResSys &s, int mixed, double eps_inner, unsigned rank, unsigned nb,
                                          double *sm, ResShared *sh) {
  if (test_skip_barrier(s.sc, rank)) {  // a lone CTA has no partner whose wait could run out
    if (nb == 1 && threadIdx.x == 0) set_status(s.sc, FREHD_ERR_TIMEOUT);
    return false;
  }
  if (kMix && mixed) {
    const int r = res_mixed<KR>(s, eps_inner, rank, nb, sm, sh);
    if (r != 2) return r == 1;
    const bool ok = res_fp64<KR>(s, rank, nb, sm, sh);
    if (ok && rank == 0 && threadIdx.x == 0) s.sc->cg_fallback = 2;
    return ok;
  }
  return res_fp64<KR>(s, rank, nb, sm, sh);
}

}  // namespace

template <int KR, bool kMix>
__global__ void __launch_bounds__(kCgThreads, 1) k_cgr(View w, int x0_surface, int eliminate) {
  if (*(volatile int *)&w.sc->status != FREHD_OK) return;
  extern __shared__ __align__(16) double res_sm[];
  __shared__ ResShared sh;
  ResSys s;
  sys_of(w, x0_surface, eliminate, &s);
  res_solve<KR, kMix>(s, w.p.mixed, w.p.eps_inner, blockIdx.x, gridDim.x, res_sm, &sh);
}

template <bool kMix>
__global__ void __launch_bounds__(kCgThreads, 1)
    k_cgr_batch(const View *__restrict__ views2, const int *__restrict__ job_start,
                const CgJob *__restrict__ jobs, const CgJob *__restrict__ singles, int nsingles, int *taken) {
  extern __shared__ __align__(16) double res_sm[];
  __shared__ ResShared sh;
  __shared__ ResSys s_sys;
  __shared__ double s_eps;
  __shared__ int s_mixed, s_next, s_run;
  const int q0 = job_start[blockIdx.x], nstatic = job_start[blockIdx.x + 1] - q0;
  for (int n = 0;; ++n) {
    CgJob jb;
    if (n < nstatic) {
      jb = jobs[q0 + n];
    } else {
      __syncthreads();  // every thread read the previous s_next
      if (threadIdx.x == 0) s_next = atomicAdd(taken, 1);
      __syncthreads();
      if (s_next >= nsingles) break;
      jb = singles[s_next];
    }
    __syncthreads();  // the previous job is done with the shared system
    if (threadIdx.x == 0) {
      const View *v = views2 + 2 * jb.d;
      v += *(volatile int *)&v->sc->cur;
      sys_of(*v, jb.flags & 1, (jb.flags >> 1) & 1, &s_sys);
      s_mixed = v->p.mixed;
      s_eps = v->p.eps_inner;
      s_run = *(volatile int *)&v->sc->status == FREHD_OK;
    }
    __syncthreads();
    if (!s_run) continue;
    // a solve that gave up has marked its own domain; the CTA goes on with the next
    switch (jb.flags >> 4) {
      case 1: res_solve<1, kMix>(s_sys, s_mixed, s_eps, jb.rank, jb.nb, res_sm, &sh); break;
      case 2: res_solve<2, kMix>(s_sys, s_mixed, s_eps, jb.rank, jb.nb, res_sm, &sh); break;
      default: res_solve<4, kMix>(s_sys, s_mixed, s_eps, jb.rank, jb.nb, res_sm, &sh); break;
    }
  }
}

// ---------------------------------------------------------------- host side

namespace {

void *single_fn(int rows, bool mix) {
  switch (rows) {
    case 1: return mix ? (void *)k_cgr<1, true> : (void *)k_cgr<1, false>;
    case 2: return mix ? (void *)k_cgr<2, true> : (void *)k_cgr<2, false>;
    default: return mix ? (void *)k_cgr<4, true> : (void *)k_cgr<4, false>;
  }
}
void *batch_fn(bool mix) { return mix ? (void *)k_cgr_batch<true> : (void *)k_cgr_batch<false>; }

}  // namespace

int cgr_capacity(int device, int *ctas) {
  int nsm = 0, least = 1 << 30;
  cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  auto one = [&](void *fn, unsigned smem) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kCgThreads, smem);
    if (per < least) least = per;
  };
  for (int mix = 0; mix < 2; ++mix) {
    for (int rows = 1; rows <= kResMaxKR; rows *= 2) one(single_fn(rows, mix), res_smem(rows));
    one(batch_fn(mix), res_smem(kResMaxKR));
  }
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "resident solve set-up: %s", cudaGetErrorString(e));
  if (least < 1) return fail(FREHD_ERR_CUDA, "the resident solve does not fit on an SM");
  *ctas = nsm;  // one CTA per SM: more would share the SM's latency, not hide it
  return FREHD_OK;
}

long long cgr_exchange_bytes(const Grid &g, int rows) {
  long n = 0;  // a batch may take more rows per thread
  for (int KR = rows; KR && KR <= kResMaxKR; KR *= 2) {
    const long e = res_entries(res_tiles(g.nx, g.ny, KR), KR);
    if (e > n) n = e;
  }
  return 16LL * n;
}

int cgr_launch(const View &w, int rows, int x0_surface, int eliminate, cudaStream_t stream) {
  View wv = w;
  int x0 = x0_surface, el = eliminate;
  void *args[] = {&wv, &x0, &el};
  const long nb = res_tiles(w.gr.nx, w.gr.ny, rows);
  cudaError_t e = cudaLaunchCooperativeKernel(single_fn(rows, w.p.mixed != 0), dim3((unsigned)nb), dim3(kCgThreads),
                                              args, res_smem(rows), stream);
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "k_cgr launch: %s", cudaGetErrorString(e));
  return FREHD_OK;
}

int cgr_launch_batch(const View *views2, const int *job_start, const CgJob *jobs, const CgJob *singles,
                     int nsingles, int *taken, int nctas, int any_mixed, cudaStream_t stream) {
  void *args[] = {&views2, &job_start, &jobs, &singles, &nsingles, &taken};
  cudaError_t e = cudaLaunchCooperativeKernel(batch_fn(any_mixed != 0), dim3(nctas), dim3(kCgThreads), args,
                                              res_smem(kResMaxKR), stream);
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "k_cgr_batch launch: %s", cudaGetErrorString(e));
  return FREHD_OK;
}

}  // namespace frehd
