// Kernels of the resident solve (cg_res.cuh): one domain, or many in a batch.
#include "cg_res.cuh"

#include <mutex>

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
  s->beat = nullptr;
}

// A batched solve's CTAs come to it one by one, each from solves of its own, and a
// partner may be held up for as long as those take: hundreds of thousands of iterations,
// or the whole wait of one that gives up.  None of that is this domain's time-out, so
// its solve starts, and its waits count, once all nb CTAs are there.  That wait ends too:
// it gives up when no solve of the launch has shown a sign of life (a solve that ends,
// or kResBeat reductions) for several times the longest that a solve waits in vain.
// (The caller has counted itself in.)
__device__ __forceinline__ bool res_all_here(Scratch *sc, unsigned nb, unsigned *beat) {
  volatile unsigned *arrived = &sc->res_arrived;
  volatile int *status = &sc->status;
  for (int n = 0; n < 64; ++n) {  // (both on their way together, and nothing else)
    const unsigned here = *arrived;
    const int st = *status;
    if (st != FREHD_OK) return false;
    if (here >= nb) return true;
  }
  const unsigned long long own = sc->wait_limit_ns;
  const unsigned long long lim = 5 * (own > kBarrierTimeoutNs ? own : kBarrierTimeoutNs);
  unsigned seen = *(volatile unsigned *)beat;
  unsigned long long t0 = gtimer_ns();
  for (;;) {
    const unsigned here = *arrived, now = *(volatile unsigned *)beat;
    if (*status != FREHD_OK) return false;
    if (here >= nb) return true;
    if (now != seen) {
      seen = now;
      t0 = gtimer_ns();
    } else if (gtimer_ns() - t0 > lim) {
      set_status(sc, FREHD_ERR_TIMEOUT);
      return false;
    }
  }
}

// The two solves as functions of their own: in one kernel with each other or with
// other tile heights they must not share a register allocation (the inlined FP32
// sweeps of 64 x 64 tiles spilled 2.6 KB).
template <int KR, bool kBatch>
__device__ __noinline__ ResEnd res_job_mixed(const ResSys *sp, double eps_inner, unsigned rank, unsigned nb,
                                          unsigned csize) {
  extern __shared__ __align__(16) double res_sm[];
  __shared__ ResShared sh;
  const ResSys s = *sp;
  return res_mixed<KR, kBatch>(s, eps_inner, rank, nb, csize, res_sm, &sh);
}
template <int KR, bool kBatch>
__device__ __noinline__ bool res_job_fp64(const ResSys *sp, unsigned rank, unsigned nb, unsigned csize,
                                          unsigned from) {
  extern __shared__ __align__(16) double res_sm[];
  __shared__ ResShared sh;
  const ResSys s = *sp;
  return res_fp64<KR, kBatch>(s, rank, nb, csize, from, res_sm, &sh);
}

// The domain's solve in its configured precision by nb CTAs (in clusters of csize); sp
// in shared memory.  kAlone: the FP64 solve is the kernel's only one (inlined: 4.56 us
// per iteration at 512 x 512 against 5.39).
template <int KR, bool kMix, bool kAlone, bool kBatch>
__device__ __forceinline__ void res_solve(const ResSys *sp, int mixed, double eps_inner, unsigned rank, unsigned nb,
                                          unsigned csize) {
  if (test_skip_barrier(sp->sc, rank)) {  // a lone CTA has no partner whose wait could run out
    if (nb == 1 && threadIdx.x == 0) set_status(sp->sc, FREHD_ERR_TIMEOUT);
    return;
  }
  if (kMix && mixed) {
    const ResEnd end = res_job_mixed<KR, kBatch>(sp, eps_inner, rank, nb, csize);
    if (end.code != 2) return;
    if (res_job_fp64<KR, kBatch>(sp, rank, nb, csize, end.tag) && rank == 0 && threadIdx.x == 0) sp->sc->cg_fallback = 2;
    return;
  }
  if (kAlone) {
    extern __shared__ __align__(16) double res_sm[];
    __shared__ ResShared sh;
    const ResSys s = *sp;
    res_fp64<KR, kBatch>(s, rank, nb, csize, 0, res_sm, &sh);
  } else {
    res_job_fp64<KR, kBatch>(sp, rank, nb, csize, 0);
  }
}

}  // namespace

// Whether this launch stands in clusters of csize, block b being CTA b % csize of its
// own: as the hardware says, whatever the launch asked for.  (A profiler's replay of a
// cooperative launch in clusters may come without them, and a store to a CTA that the
// cluster does not have is a fault.)
__device__ __forceinline__ bool res_in_clusters(int csize) {
  unsigned n, rank;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return n == (unsigned)csize && rank == blockIdx.x % csize;
}

// nb CTAs solve; the grid is a multiple of the cluster size csize, and the CTAs past
// nb only keep their clusters whole.  Without the clusters all entries go through L2
// (the same sums).  fill(&s): the system, by one thread.
template <int KR, bool kMix, class F>
__device__ __forceinline__ void res_kernel(Scratch *sc, int mixed, double eps_inner, int nb, int csize, F fill) {
  extern __shared__ __align__(16) double res_sm[];
  __shared__ ResSys s;
  __shared__ int s_run;
  if (csize > 1 && !res_in_clusters(csize)) csize = 1;
  if (csize > 1) {
    // the inbox carries no tag before a neighbour may write to it
    uint4 *in = reinterpret_cast<uint4 *>(res_sm + kResSums * kResThreads + 3 * res_arr(KR));
    for (int e = threadIdx.x; e < res_inbox(KR); e += kResThreads) in[e] = make_uint4(0, 0, 0, 0);
    res_cluster_sync();
  }
  // (a step that has failed is skipped, but no CTA leaves its cluster early; one thread
  // looks, since another CTA of this solve may set the status meanwhile)
  if (threadIdx.x == 0) {
    s_run = (int)blockIdx.x < nb && *(volatile int *)&sc->status == FREHD_OK;
    if (s_run) fill(&s);
  }
  __syncthreads();
  if (s_run) res_solve<KR, kMix, !kMix, false>(&s, mixed, eps_inner, blockIdx.x, nb, csize);
  // no store into this CTA's shared memory is on its way any more
  if (csize > 1) res_cluster_sync();
}

template <int KR, bool kMix>
__global__ void __launch_bounds__(kResThreads, 1) k_cgr(View w, int x0_surface, int eliminate, int nb, int csize) {
  res_kernel<KR, kMix>(w.sc, w.p.mixed, w.p.eps_inner, nb, csize,
                       [&](ResSys *s) { sys_of(w, x0_surface, eliminate, s); });
}

template <int KR>
__global__ void __launch_bounds__(kResThreads, 1) k_cgr_sys(ResSys sys, int nb, int csize) {
  res_kernel<KR, false>(sys.sc, 0, 0.0, nb, csize, [&](ResSys *s) { *s = sys; });
}

template <bool kMix>
__global__ void __launch_bounds__(kResThreads, 1)
    k_cgr_batch(const View *__restrict__ views2, const int *__restrict__ job_start,
                const CgJob *__restrict__ jobs, const CgJob *__restrict__ singles, int nsingles, Scratch *bsync) {
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
      if (threadIdx.x == 0) s_next = atomicAdd(&bsync->taken, 1);
      __syncthreads();
      if (s_next >= nsingles) break;
      jb = singles[s_next];
    }
    __syncthreads();  // the previous job is done with the shared system
    if (threadIdx.x == 0) {
      const View *v = views2 + 2 * jb.d;
      Scratch *sc = v->sc;
      atomicAdd(&sc->res_arrived, 1u);
      v += *(volatile int *)&sc->cur;
      sys_of(*v, jb.flags & 1, (jb.flags >> 1) & 1, &s_sys);
      s_sys.beat = &bsync->beat;
      s_mixed = v->p.mixed;
      s_eps = v->p.eps_inner;
      s_run = res_all_here(sc, jb.nb, &bsync->beat);
    }
    __syncthreads();
    if (!s_run) continue;
    // a solve that gave up has marked its own domain; the CTA goes on with the next
    switch (jb.flags >> 4) {
      case 1: res_solve<1, kMix, false, true>(&s_sys, s_mixed, s_eps, jb.rank, jb.nb, 1); break;
      case 2: res_solve<2, kMix, false, true>(&s_sys, s_mixed, s_eps, jb.rank, jb.nb, 1); break;
      default: res_solve<4, kMix, false, true>(&s_sys, s_mixed, s_eps, jb.rank, jb.nb, 1); break;
    }
    if (threadIdx.x == 0) atomicAdd(&bsync->beat, 1u);
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
void *sys_fn(int rows) {
  switch (rows) {
    case 1: return (void *)k_cgr_sys<1>;
    case 2: return (void *)k_cgr_sys<2>;
    default: return (void *)k_cgr_sys<4>;
  }
}
void *batch_fn(bool mix) { return mix ? (void *)k_cgr_batch<true> : (void *)k_cgr_batch<false>; }

}  // namespace

namespace {

// Clusters of `size` CTAs of kernel fn that the device holds at once (0: none).
int max_clusters(void *fn, unsigned smem, int size) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace

int cgr_capacity(int device, int *ctas, int *clustered) {
  // found once per device; domains may be created on several host threads
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static struct {
    int ctas, clustered;
  } known[kMaxDevices];
  std::lock_guard<std::mutex> lk(mu);
  if (device >= 0 && device < kMaxDevices && known[device].ctas) {
    *ctas = known[device].ctas;
    *clustered = known[device].clustered;
    return FREHD_OK;
  }
  int nsm = 0, least = 1 << 30, clustered_n = kResClustered;
  cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  auto one = [&](void *fn, unsigned smem, bool in_clusters) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kResThreads, smem);
    if (per < least) least = per;
    if (!in_clusters || e != cudaSuccess) return;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return;
    // as many CTAs as every form of cluster below that count allows
    int n = max_clusters(fn, smem, kResFlat) < 1 ? 0 : 4 * max_clusters(fn, smem, 4);
    if (8 * max_clusters(fn, smem, 8) < kResEights) n = n < kResFlat ? n : kResFlat;
    if (n < clustered_n) clustered_n = n;
  };
  for (int rows = kResMinKR; rows <= kResMaxKR; rows *= 2) one(sys_fn(rows), res_smem(rows), true);
  for (int mix = 0; mix < 2; ++mix) {
    for (int rows = kResMinKR; rows <= kResMaxKR; rows *= 2) one(single_fn(rows, mix), res_smem(rows), true);
    one(batch_fn(mix), res_smem(kResMaxKR), false);
  }
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "resident solve set-up: %s", cudaGetErrorString(e));
  if (least < 1) return fail(FREHD_ERR_CUDA, "the resident solve does not fit on an SM");
  *ctas = nsm;  // one CTA per SM: more would share the SM's latency, not hide it
  *clustered = clustered_n;
  if (device >= 0 && device < kMaxDevices) known[device] = {*ctas, *clustered};
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

namespace {

// Kernel fn on the nb tiles of a solve, cooperatively and, where that fits, in clusters
// (own: pointers to the kernel's own arguments; nb and the cluster size follow them).
// plain: the clusters are announced to the kernel but not asked for.
template <int N>
int launch_solve(void *fn, void *const (&own)[N], int nx, int ny, int rows, int clustered, bool plain,
                 cudaStream_t stream) {
  int nb = (int)res_tiles(nx, ny, rows), csize = nb <= kResFlat ? nb : res_group(nb);
  if (nb > clustered) csize = 1;
  void *args[N + 2];
  for (int n = 0; n < N; ++n) args[n] = own[n];
  args[N] = &nb;
  args[N + 1] = &csize;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = csize;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((nb + csize - 1) / csize * csize));
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = res_smem(rows);
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = csize > 1 && !plain ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "resident solve launch: %s", cudaGetErrorString(e));
  return FREHD_OK;
}

}  // namespace

int cgr_launch(const View &w, int rows, int clustered, bool plain, int x0_surface, int eliminate,
               cudaStream_t stream) {
  View wv = w;
  void *const own[] = {&wv, &x0_surface, &eliminate};
  return launch_solve(single_fn(rows, w.p.mixed != 0), own, w.gr.nx, w.gr.ny, rows, clustered, plain,
                      stream);
}

int cgr_launch_sys(const ResSys &s, int rows, int clustered, cudaStream_t stream) {
  ResSys sv = s;
  void *const own[] = {&sv};
  return launch_solve(sys_fn(rows), own, s.nx, s.ny, rows, clustered, false, stream);
}

int cgr_launch_batch(const View *views2, const int *job_start, const CgJob *jobs, const CgJob *singles,
                     int nsingles, Scratch *bsync, int nctas, int any_mixed, cudaStream_t stream) {
  void *args[] = {&views2, &job_start, &jobs, &singles, &nsingles, &bsync};
  cudaError_t e = cudaLaunchCooperativeKernel(batch_fn(any_mixed != 0), dim3(nctas), dim3(kResThreads), args,
                                              res_smem(kResMaxKR), stream);
  if (e != cudaSuccess) return fail(FREHD_ERR_CUDA, "k_cgr_batch launch: %s", cudaGetErrorString(e));
  return FREHD_OK;
}

}  // namespace frehd
