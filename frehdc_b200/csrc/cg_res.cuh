// Resident Jacobi-PCG: the single-sweep solve of cg1.cu (same scaled system,
// same recurrences, same stopping rule and fall-back) for domains whose solver
// state fits on chip.
//
// What bounds a small solve is not traffic but the latency of an iteration: with
// the state in HBM every iteration waits for its TMA boxes and for a two-hop
// grid reduction (arrive, last block sums and publishes, everyone reads), 11 us
// per iteration at 128 x 128.  Here each CTA keeps one tile of
// 64 x (16 KR) cells for the whole solve: vectors and couplings in registers, with
// a copy of the residual in shared memory where the stencil's neighbours read it.
// An iteration then touches global memory twice, both in one hop:
//   * the tile's outer second row and column of the new residual (what a
//     neighbour tile cannot compute itself: it recomputes the first ring), and
//   * the CTA's six partial sums, added in an order fixed by the ranks.
// Both travel as 16-byte entries {low word, tag, high word, tag}, the layout and the one
// 16-byte access of NCCL's LL protocol: the tag is the reduction's number, so an entry
// announces itself and neither a fence nor an arrival counter stands between the
// writer's store and the reader's load.  (An entry orders itself only: where other
// memory is to be read after a reduction, res_exchange fences.)  The
// entries alternate between two buffers by tag parity; no CTA can write the
// buffer of reduction t + 2 before every CTA has published t + 1, that is,
// finished reading t.
//
// The CTAs of one solve form clusters: of all of them up to kResFlat, of res_group up
// to kResClustered (more do not fit the device in clusters).  Inside a cluster an entry
// is stored straight into its reader's shared memory, where polling costs nothing
// (through L2 every reader polls the line that its writer is waiting to store: 2.4 us a
// reduction among 16 CTAs).  Only the
// groups' sums and the edges between clusters go through L2.  In a batch, whose CTAs
// take one solve after another in ever new groups, all entries do; the sums are added
// in the same order either way.
//
// What is left is one warp's chain of dependent instructions, about nine cycles
// each, so the FP64 iteration is arranged to be short: with w = A~ r~ from the last
// sweep, A~ p_i = w_i + beta A~ p_{i-1} needs no second stencil (it holds for any
// A~), the first ring's w is formed while the sums travel, the sums themselves
// go through shared memory to one warp per sum, and only the stencil of the new
// residual and two barriers lie between the scalars and the sums.  The FP32 inner
// sweep of the mixed solve keeps the two stencils of sweep() in cg1.cu, rounding for
// rounding.
//
// Tags only grow: a launch starts at Scratch::res_tag, and every CTA raises it
// to the last tag it used, whether it ends well or after a wait that gave up.  Near
// their end a solve clears the entries and starts them again (res_enter).
//
// Rounding: A p by its recurrence and the scaling by sqrt|Ct| are as good as the stencil
// on p and the unscaled system while a solve takes hundreds of iterations (the error
// against 64-bit references is the same to two digits up to 300, and to 2000 at
// tolerances above 1e-13).  Past that, where a tolerance asks for all the digits that a
// condition number near 1e7 and more leaves, the solution attained is further off:
// 2e-14 against 8e-15 after 1000 iterations, 2e-11 against 2e-13 after 7400 (couplings
// over six decades); the scaling, which k_cg1 has too, is most of it.
#ifndef FREHD_CG_RES_CUH
#define FREHD_CG_RES_CUH

#include "cg_common.cuh"
#include "cg_limit.h"
#include "cg_res.h"

namespace frehd {

struct ResShared {
  double tot[kResSlot];
  double scale, inv_gamma;  // 1 / (scale gamma) of the last sweep (res_keep)
  unsigned tag;    // the tag the solve starts from
  unsigned *beat;  // ResSys::beat (batched solves)
  int ok;
};

// Where a CTA stands: its rank among the nb of the solve, the tag of the last
// reduction, and the buffers.
struct ResCtx {
  unsigned rank, nb, tag;
  unsigned csize;  // CTAs of a cluster (1: none, entries go through L2)
  unsigned inbox;  // this CTA's inbox, as a shared-memory address
  uint4 *slots, *edges;
  Scratch *sc;
  ResShared *sh;
  double *sums;  // kResSums x kResThreads in shared memory
};


namespace {

// From this tag on a solve first clears its entries and starts again at 0: a quarter of
// the numbers are left for the reductions of that solve's launch.
constexpr unsigned kResTagEnd = 0xC0000000u;
// Reductions between two signs of life of a solve (a few milliseconds).
constexpr unsigned kResBeat = 1024;

__device__ __forceinline__ uint4 res_ld(const uint4 *a) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void res_st(uint4 *a, double d, unsigned tag) {
  const unsigned long long q = (unsigned long long)__double_as_longlong(d);
  asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(a), "r"((unsigned)q), "r"(tag),
               "r"((unsigned)(q >> 32)), "r"(tag)
               : "memory");
}
__device__ __forceinline__ double res_val(const uint4 &v) {
  return __longlong_as_double((long long)(((unsigned long long)v.z << 32) | v.x));
}

// An entry in another CTA's shared memory (address res_at) or in one's own.
__device__ __forceinline__ unsigned res_at(unsigned addr, unsigned cta) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void res_sts(unsigned at, double d, unsigned tag) {
  const unsigned long long q = (unsigned long long)__double_as_longlong(d);
  asm volatile("st.relaxed.cluster.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"((unsigned)q),
               "r"(tag), "r"((unsigned)(q >> 32)), "r"(tag)
               : "memory");
}
__device__ __forceinline__ uint4 res_lds(unsigned addr) {
  uint4 v;
  asm volatile("ld.relaxed.cluster.shared::cta.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void res_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// The entry each lane loads (if it has one), once all of the warp's carry `tag`: by
// the whole warp, in step.  A warp whose lanes left a polling loop one by one would
// issue what follows once per lane (1300 cycles for the five shuffles of a sum).
// The first polls look at nothing else (reading the clock or the limit costs as long as
// the wait itself); after that the wait is bounded (ok becomes 0).
template <class L>
__device__ __forceinline__ double res_wait(bool has, L load, unsigned tag, Scratch *sc, int *ok) {
  uint4 e = make_uint4(0, tag, 0, tag);
#pragma unroll 1
  for (int n = 0; n < 2048; ++n) {
    if (has) e = load();
    if (__all_sync(0xffffffffu, e.y == tag && e.w == tag)) return res_val(e);
  }
  const unsigned long long lim = sc->wait_limit_ns ? sc->wait_limit_ns : kBarrierTimeoutNs;
  const unsigned long long t0 = gtimer_ns();
#pragma unroll 1
  for (;;) {
    if (has) e = load();
    if (__all_sync(0xffffffffu, e.y == tag && e.w == tag)) return res_val(e);
    const bool over = *(volatile int *)&sc->status == FREHD_ERR_TIMEOUT || gtimer_ns() - t0 > lim;
    if (__any_sync(0xffffffffu, over)) {
      set_status(sc, FREHD_ERR_TIMEOUT);
      *(volatile int *)ok = 0;
      return 0.0;
    }
  }
}

__device__ __forceinline__ double res_warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Inbox entries (parity, value m): rank r's sum in the cluster, the total.
__device__ __forceinline__ unsigned res_in_sum(const ResCtx &c, int m, unsigned r) {
  return c.inbox + 16u * (((c.tag & 1) * kResSlot + m) * (kResFlat + 1) + r);
}
__device__ __forceinline__ unsigned res_in_total(const ResCtx &c, int m) { return res_in_sum(c, m, kResFlat); }
template <int KR>
__device__ __forceinline__ unsigned res_in_edge(const ResCtx &c, unsigned tag, int e) {
  return c.inbox + 16u * (2 * kResSlot * (kResFlat + 1) + (tag & 1) * res_edge(KR) + e);
}

// Entries in L2 (parity, value m): a rank's sum, a group's; one value's lie together, so
// that a warp's poll touches few lines.
__device__ __forceinline__ uint4 *res_slot(const ResCtx &c, unsigned rank, int m) {
  return c.slots + ((c.tag & 1) * kResSlot + m) * c.nb + rank;
}
__device__ __forceinline__ uint4 *res_top(const ResCtx &c, unsigned g, int m) {
  return c.slots + 2L * c.nb * kResSlot + ((c.tag & 1) * kResSlot + m) * kResMaxGroups + g;
}

// Between what a warp's lanes have read and what any of them passes on.
__device__ __forceinline__ void res_relay_fence() {
  __threadfence();
  __syncwarp();
  __threadfence();
}

// The CTAs' sums t of value m, added up: by the whole of one warp, the same total in
// every CTA.  Up to kResFlat CTAs in one tree over the ranks, else by groups of
// res_group(nb) and then over the groups.
// kFence: what the CTAs' threads stored in global memory before the reduction is to be
// read after it.  The entries themselves order nothing, so the warp that sends them
// fences after the block barrier in front, the relays between reading and passing on,
// and every warp after its last read.
template <bool kFence>
__device__ __forceinline__ double res_exchange(double t, int m, const ResCtx &c) {
  const unsigned lane = threadIdx.x & 31;
  int *ok = &c.sh->ok;
  if (kFence) __threadfence();
  if (c.nb <= (unsigned)kResFlat) {
    if (c.csize > 1) {
      if (lane < c.nb) res_sts(res_at(res_in_sum(c, m, c.rank), lane), t, c.tag);
      t = res_wait(lane < c.nb, [&] { return res_lds(res_in_sum(c, m, lane)); }, c.tag, c.sc, ok);
    } else {
      if (lane == 0) res_st(res_slot(c, c.rank, m), t, c.tag);
      t = res_wait(lane < c.nb, [&] { return res_ld(res_slot(c, lane, m)); }, c.tag, c.sc, ok);
    }
    if (kFence) __threadfence();
    return res_warp_total(t);
  }
  const unsigned group = res_group(c.nb), groups = (c.nb + group - 1) / group;
  if (c.csize > 1) {
    const unsigned mine = c.rank % group, g = c.rank / group, members = min(group, c.nb - g * group);
    if (mine) {  // to the group's first CTA, and the total back
      if (lane == 0) res_sts(res_at(res_in_sum(c, m, mine), 0), t, c.tag);
      t = res_wait(true, [&] { return res_lds(res_in_total(c, m)); }, c.tag, c.sc, ok);
      if (kFence) __threadfence();
      return t;
    }
    const double own = t;
    t = res_wait(lane > 0 && lane < members, [&] { return res_lds(res_in_sum(c, m, lane)); }, c.tag, c.sc, ok);
    t = res_warp_total(lane == 0 ? own : t);
    if (kFence) res_relay_fence();
    if (lane == 0) res_st(res_top(c, g, m), t, c.tag);
    t = res_wait(lane < groups, [&] { return res_ld(res_top(c, lane, m)); }, c.tag, c.sc, ok);
    t = res_warp_total(t);
    if (kFence) res_relay_fence();
    if (lane > 0 && lane < members) res_sts(res_at(res_in_total(c, m), lane), t, c.tag);
    return t;
  }
  if (lane == 0) res_st(res_slot(c, c.rank, m), t, c.tag);
  // 32 ranks at a time, the next 32 on their way meanwhile; the groups' trees run side by
  // side in the lanes (past kResClustered CTAs there are more groups than lanes: the
  // ranks in one tree)
  const bool grouped = c.nb <= (unsigned)kResClustered;
  t = 0.0;
  uint4 next = make_uint4(0, 0, 0, 0);
#pragma unroll 1
  for (unsigned r0 = 0; r0 < c.nb; r0 += 32) {
    const bool has = r0 + lane < c.nb, first = r0 == 0;
    const uint4 early = next;
    if (r0 + 32 + lane < c.nb) next = res_ld(res_slot(c, r0 + 32 + lane, m));
    double v = 0.0;
    if (!first && __all_sync(0xffffffffu, !has || (early.y == c.tag && early.w == c.tag)))
      v = has ? res_val(early) : 0.0;
    else
      v = res_wait(has, [&] { return res_ld(res_slot(c, r0 + lane, m)); }, c.tag, c.sc, ok);
    if (!grouped) {
      t += v;
      continue;
    }
#pragma unroll 1
    for (unsigned o = group / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const unsigned per = 32 / group;
    const double x = __shfl_sync(0xffffffffu, v, (lane % per) * group);
    if (lane / per == r0 / 32) t = x;
  }
  if (kFence) __threadfence();
  return res_warp_total(!grouped || lane < groups ? t : 0.0);
}

// v[0 .. NV) summed over all threads of the solve's CTAs (the same totals in each
// thread), and a barrier among them for the entries stored before it under this tag
// (the caller has advanced it).  Warp m sums value m, in the CTA and over the CTAs;
// `meanwhile` runs in the others.  False after a wait that gave up.
template <int NV, bool kFence = false, class M>
__device__ __forceinline__ bool res_allreduce(double (&v)[kResSums], const ResCtx &c, M meanwhile) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  ResShared *sh = c.sh;
#pragma unroll
  for (int m = 0; m < NV; ++m) c.sums[m * kResThreads + threadIdx.x] = v[m];
  __syncthreads();
  if (wid < NV) {
    const double2 *a = reinterpret_cast<const double2 *>(c.sums + wid * kResThreads) + lane;
    double part[kResThreads / 64];
#pragma unroll
    for (int q = 0; q < kResThreads / 64; ++q) {
      const double2 e = a[32 * q];
      part[q] = e.x + e.y;
    }
#pragma unroll
    for (int n = kResThreads / 128; n > 0; n >>= 1)
#pragma unroll
      for (int q = 0; q < n; ++q) part[q] += part[q + n];
    double t = res_warp_total(part[0]);
    if (c.nb > 1) t = res_exchange<kFence>(t, wid, c);
    if (lane == 0) sh->tot[wid] = t;
  } else {
    meanwhile();
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < NV; ++m) v[m] = sh->tot[m];
  return *(volatile int *)&sh->ok;
}

template <typename T>
struct ResPair;
template <>
struct ResPair<double> {
  using type = double2;
};
template <>
struct ResPair<float> {
  using type = float2;
};

// A thread's part of the tile: KR rows of two cells, and at most one cell of the
// first ring around the tile (the last warps have them, the first ones the sums).
// The ring cell's outer neighbour (and, at the end of a side, the diagonal one)
// lies in a neighbour tile, which publishes its residual; the thread likewise
// publishes one cell of its own tile.
template <typename T, int KR>
struct ResTile {
  T r[KR][2], p[KR][2], x[KR][2];
  T hx[KR][3], hy[KR + 1][2];  // couplings of the rows' x faces (west, middle, east) and y faces
  T r1, h1[4], r2[2];          // ring cell; couplings east, west, north, south; outer and diagonal
  unsigned dec;                // bit 2k + c: decoupled cell; bit 31: decoupled ring cell
  int q1;                      // shared-memory position of the ring cell (-1: none)
  int dir;                     // direction of the outer neighbour, and 4 x that of the diagonal one
  const uint4 *src[2];         // their exchange entries (parity 0) in L2, or null,
  int in[2];                   // or their number in the inbox, or -1 (neither: outside the domain)
  int qp;                      // shared-memory position of the cell to publish (-1: none)
  uint4 *dst;                  // its exchange entry (parity 0) in L2, or null and
  unsigned out[2];             // its address in the neighbour's inbox, by parity
};

// Ring cell e: its tile coordinates, the direction of its outer neighbour (0 east,
// 1 west, 2 north, 3 south) and of the diagonal cell beside it (4: none).
template <int KR>
__device__ __forceinline__ bool res_ring(int e, int *lx, int *ly, int *outer, int *diag) {
  constexpr int TH = res_th(KR), TW = kResTW;
  *diag = 4;
  if (e < 2 * TW) {
    *outer = e < TW ? 3 : 2;
    *ly = e < TW ? -1 : TH;
    *lx = e < TW ? e : e - TW;
    if (*lx == 0) *diag = 1;
    if (*lx == TW - 1) *diag = 0;
    return true;
  }
  e -= 2 * TW;
  *outer = e < TH ? 1 : 0;
  *lx = e < TH ? -1 : TW;
  *ly = e < TH ? e : e - TH;
  if (*ly == 0) *diag = 3;
  if (*ly == TH - 1) *diag = 2;
  return e < 2 * TH;
}

// The tile (dx, dy) beside this one that owns cell (lx, ly) two cells out or
// diagonally off a corner, and the cell's exchange entry there: west column | east
// column | south row | north row | corners south-west, south-east, north-west,
// north-east.
template <int KR>
__device__ __forceinline__ int res_owner(int lx, int ly, int *dx, int *dy) {
  constexpr int TH = res_th(KR), TW = kResTW;
  *dx = lx < 0 ? -1 : (lx >= TW ? 1 : 0);
  *dy = ly < 0 ? -1 : (ly >= TH ? 1 : 0);
  if (*dx && *dy)  // my south-west diagonal cell is that tile's north-east corner, and so on
    return 2 * TH + 2 * TW + (*dy < 0 ? 2 : 0) + (*dx < 0 ? 1 : 0);
  if (*dy) return 2 * TH + lx + (*dy < 0 ? TW : 0);
  return ly + (*dx < 0 ? TH : 0);
}

__device__ __forceinline__ int res_step(int dir) {
  return dir == 0 ? 1 : dir == 1 ? -1 : dir == 2 ? kResPitch : -kResPitch;
}

__device__ __forceinline__ int res_q(int lx, int ly) { return (ly + 2) * kResPitch + lx + 2; }

__device__ __forceinline__ bool res_in(const ResSys &s, int i, int j) {
  return (unsigned)i < (unsigned)s.nx && (unsigned)j < (unsigned)s.ny;
}

// r = b - A x at cell (i, j) of the interior, x given by xat(k); with elim the
// decoupled neighbours stand at their exact b/|Ct|.
template <class X>
__device__ __forceinline__ double res_residual(const ResSys &s, int i, int j, int elim, X xat) {
  const long k = s.off + (long)j * s.pitch + i;
  const double ct = s.Ct[k], bk = s.b[k], xk = xat(k);
  if (!(ct > 0)) return bk - (-ct) * xk;
  auto xv = [&](bool in, long kk) -> double {
    if (!in) return 0.0;
    const double cc = s.Ct[kk];
    return (elim && cc < 0) ? s.b[kk] / (-cc) : xat(kk);
  };
  const double ge = i + 1 < s.nx ? s.Gx[k] : 0.0, gw = i > 0 ? s.Gx[k - 1] : 0.0;
  const double gn = j + 1 < s.ny ? s.Gy[k] : 0.0, gs = j > 0 ? s.Gy[k - s.pitch] : 0.0;
  const double ax = ct * xk - (ge * xv(i + 1 < s.nx, k + 1) + gw * xv(i > 0, k - 1) +
                               gn * xv(j + 1 < s.ny, k + s.pitch) + gs * xv(j > 0, k - s.pitch));
  return bk - ax;
}

// The same of an x in global memory (L2) and the padded layout of a domain, whose
// ghost ring stands for the cells outside (couplings 0 there).  The roundings are
// spelled out: a closed dry cell's x ends within an ulp of its bed, and on which
// side decides the limiter, so this pass and cg1_mixed's round alike.
__device__ __forceinline__ double res_residual_padded(const ResSys &s, const double *X, int i, int j, int elim) {
  const long k = s.off + (long)j * s.pitch + i;
  const double ct = s.Ct[k], bk = s.b[k], xk = __ldcg(X + k);
  if (!(ct > 0)) return fma(ct, xk, bk);
  auto xv = [&](long kk) -> double {
    const double cc = s.Ct[kk];
    return (elim && cc < 0) ? s.b[kk] / (-cc) : __ldcg(X + kk);
  };
  double ax = __dmul_rn(s.Gx[k], xv(k + 1));
  ax = fma(s.Gx[k - 1], xv(k - 1), ax);
  ax = fma(s.Gy[k], xv(k + s.pitch), ax);
  ax = fma(s.Gy[k - s.pitch], xv(k - s.pitch), ax);
  return __dsub_rn(bk, fma(ct, xk, -ax));
}

// The tile's couplings (scaled), decoupled flags and ring bookkeeping, by way
// of three shared arrays (loops over the tile and its rings: unrolled per thread,
// the divisions alone were 30 KB of code that every solve fetched anew).
template <typename T, int KR>
__device__ __forceinline__ void res_setup(const ResSys &s, const ResCtx &c, int i0, int j0, int elim,
                                          double *ds, ResTile<T, KR> &t) {
  constexpr int TH = res_th(KR), kArr = res_arr(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx), nty = (s.ny + TH - 1) / TH;
  double *dx_ = ds + kArr, *dy_ = dx_ + kArr;
  __syncthreads();
  // sqrt|Ct|, negative on decoupled rows and outside
#pragma unroll 1
  for (int e = threadIdx.x; e < kArr; e += kResThreads) {
    const int i = i0 + e % kResPitch - 2, j = j0 + e / kResPitch - 2;
    double d = -1.0;
    if (res_in(s, i, j)) {
      const double ct = s.Ct[s.off + (long)j * s.pitch + i];
      d = sqrt(fabs(ct));
      if (ct < 0) d = -d;
    }
    ds[e] = d;
  }
  __syncthreads();
  // couplings across the east and north faces
#pragma unroll 1
  for (int e = threadIdx.x; e < kArr; e += kResThreads) {
    const int cx = e % kResPitch, cy = e / kResPitch, i = i0 + cx - 2, j = j0 + cy - 2;
    double hx = 0.0, hy = 0.0;
    if (res_in(s, i, j)) {
      const long k = s.off + (long)j * s.pitch + i;
      const double a = ds[e];
      if (cx < kResPitch - 1 && i + 1 < s.nx && !(elim && !(a > 0 && ds[e + 1] > 0)))
        hx = s.Gx[k] / (fabs(a) * fabs(ds[e + 1]));
      if (cy < TH + 3 && j + 1 < s.ny && !(elim && !(a > 0 && ds[e + kResPitch] > 0)))
        hy = s.Gy[k] / (fabs(a) * fabs(ds[e + kResPitch]));
    }
    dx_[e] = hx;
    dy_[e] = hy;
  }
  __syncthreads();
  t.dec = 0;
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int q0 = res_q(2 * lane, wid * KR + k);
#pragma unroll
    for (int q = 0; q < 3; ++q) t.hx[k][q] = T(dx_[q0 + q - 1]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (k == 0) t.hy[0][q] = T(dy_[q0 + q - kResPitch]);
      t.hy[k + 1][q] = T(dy_[q0 + q]);
      if (ds[q0 + q] < 0) t.dec |= 1u << (2 * k + q);
    }
  }
  t.q1 = -1;
  t.dir = 16;
  t.src[0] = t.src[1] = nullptr;
  t.in[0] = t.in[1] = -1;
  t.r1 = t.r2[0] = t.r2[1] = T(0);
#pragma unroll
  for (int q = 0; q < 4; ++q) t.h1[q] = T(0);
  int lx, ly, outer, diag;
  const int e = kResThreads - 1 - (int)threadIdx.x;
  if (res_ring<KR>(e, &lx, &ly, &outer, &diag)) {
    t.q1 = res_q(lx, ly);
    t.h1[0] = T(dx_[t.q1]);
    t.h1[1] = T(dx_[t.q1 - 1]);
    t.h1[2] = T(dy_[t.q1]);
    t.h1[3] = T(dy_[t.q1 - kResPitch]);
    if (ds[t.q1] < 0) t.dec |= 1u << 31;
    t.dir = outer + 4 * diag;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int d = n ? diag : outer;
      if (d == 4) continue;
      int dx, dy;
      const int entry = res_owner<KR>(lx + (d == 0) - (d == 1), ly + (d == 2) - (d == 3), &dx, &dy);
      const int bx = (int)(c.rank % ntx) + dx, by = (int)(c.rank / ntx) + dy;
      if ((unsigned)bx < (unsigned)ntx && (unsigned)by < (unsigned)nty) {
        const unsigned from = (unsigned)(by * ntx + bx);
        if (c.csize > 1 && from / c.csize == c.rank / c.csize)
          t.in[n] = entry;
        else
          t.src[n] = c.edges + (long)from * 2 * res_edge(KR) + entry;
      }
    }
  }
  // exchange entry e of this tile (res_owner's order) and the tile that reads it
  t.qp = -1;
  t.dst = nullptr;
  t.out[0] = t.out[1] = 0;
  if (c.nb > 1 && e < res_edge(KR)) {
    int px, py, dx = 0, dy = 0;
    if (e < 2 * TH) {
      dx = e < TH ? -1 : 1;
      px = e < TH ? 1 : kResTW - 2;
      py = e < TH ? e : e - TH;
    } else if (e < 2 * TH + 2 * kResTW) {
      dy = e < 2 * TH + kResTW ? -1 : 1;
      px = (e - 2 * TH) % kResTW;
      py = dy < 0 ? 1 : TH - 2;
    } else {
      const int corner = e - 2 * TH - 2 * kResTW;
      dx = corner & 1 ? 1 : -1;
      dy = corner & 2 ? 1 : -1;
      px = dx > 0 ? kResTW - 1 : 0;
      py = dy > 0 ? TH - 1 : 0;
    }
    const int bx = (int)(c.rank % ntx) + dx, by = (int)(c.rank / ntx) + dy;
    const unsigned to = (unsigned)(by * ntx + bx);
    if ((unsigned)bx < (unsigned)ntx && (unsigned)by < (unsigned)nty) {
      t.qp = res_q(px, py);
      if (c.csize > 1 && to / c.csize == c.rank / c.csize) {
        for (unsigned n = 0; n < 2; ++n) t.out[n] = res_at(res_in_edge<KR>(c, n, e), to % c.csize);
      } else {
        t.dst = c.edges + (long)c.rank * 2 * res_edge(KR) + e;
      }
    }
  }
  __syncthreads();
}

// r~ (of a residual function of the interior cells) into the shared copy R of the
// tile and its rings, and from there into the tile; p = 0; adds (r~, r~) and
// ||r||^2 to acc[0], acc[1] and ||b||^2 to acc[2].  Synchronised on return.
template <typename T, int KR, class F>
__device__ __forceinline__ void res_start(const ResSys &s, int i0, int j0, T *R, ResTile<T, KR> &t,
                                          double (&acc)[kResSums], F resid) {
  constexpr int TH = res_th(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
  for (int e = threadIdx.x; e < res_arr(KR); e += kResThreads) {
    const int lx = e % kResPitch - 2, ly = e / kResPitch - 2, i = i0 + lx, j = j0 + ly;
    T rs = T(0);
    if (res_in(s, i, j)) {
      const long k = s.off + (long)j * s.pitch + i;
      const double r = resid(i, j);
      rs = T(r / sqrt(fabs(s.Ct[k])));
      if ((unsigned)lx < (unsigned)kResTW && (unsigned)ly < (unsigned)TH) {
        const double bk = s.b[k];
        acc[0] += (double)rs * (double)rs;
        acc[1] += r * r;
        acc[2] += bk * bk;
      }
    }
    R[e] = rs;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < KR; ++k)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      t.r[k][q] = R[res_q(2 * lane + q, wid * KR + k)];
      t.p[k][q] = T(0);
    }
  if (t.q1 >= 0) {
    t.r1 = R[t.q1];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int d = n ? t.dir >> 2 : t.dir & 3;
      if (d != 4) t.r2[n] = R[t.q1 + res_step(d)];
    }
  }
}

// hE E + hW W + hN N + hS S.  In FP64 as two products of two (a shorter chain); in
// FP32 in the order of apply() in cg1.cu, whose roundings the mixed solve keeps.
__device__ __forceinline__ double res_off(double he, double e, double hw, double w, double hn, double n, double hs,
                                          double s) {
  return fma(he, e, hw * w) + fma(hn, n, hs * s);
}
__device__ __forceinline__ float res_off(float he, float e, float hw, float w, float hn, float n, float hs, float s) {
  return he * e + hw * w + hn * n + hs * s;
}

// A~ v of a thread's cells (row k): v its own values; cell(q) and pair(q) give v at
// shared-memory position q (and q + 1), for the rows of other warps and the ring.
template <typename T, int KR, class C1, class C2>
__device__ __forceinline__ void res_apply(const ResTile<T, KR> &t, const T (&v)[KR][2], int k, C1 cell, C2 pair,
                                          T (&out)[2]) {
  const int lane = threadIdx.x & 31, ly = (threadIdx.x >> 5) * KR + k;
  const int q = res_q(2 * lane, ly);
  T south[2], north[2];
  if (k == 0) {
    pair(q - kResPitch, south);
  } else {
    south[0] = v[k > 0 ? k - 1 : 0][0];
    south[1] = v[k > 0 ? k - 1 : 0][1];
  }
  if (k == KR - 1) {
    pair(q + kResPitch, north);
  } else {
    north[0] = v[k < KR - 1 ? k + 1 : k][0];
    north[1] = v[k < KR - 1 ? k + 1 : k][1];
  }
  T west = __shfl_up_sync(0xffffffffu, v[k][1], 1), east = __shfl_down_sync(0xffffffffu, v[k][0], 1);
  if (lane == 0) west = cell(q - 1);
  if (lane == 31) east = cell(q + 2);
  const T off0 = res_off(t.hx[k][1], v[k][1], t.hx[k][0], west, t.hy[k + 1][0], north[0], t.hy[k][0], south[0]);
  const T off1 = res_off(t.hx[k][2], east, t.hx[k][1], v[k][0], t.hy[k + 1][1], north[1], t.hy[k][1], south[1]);
  out[0] = (t.dec >> (2 * k)) & 1u ? v[k][0] : v[k][0] - off0;
  out[1] = (t.dec >> (2 * k + 1)) & 1u ? v[k][1] : v[k][1] - off1;
}

// The same with v in the shared array V.
template <typename T, int KR>
__device__ __forceinline__ void res_apply(const ResTile<T, KR> &t, const T (&v)[KR][2], const T *V, int k,
                                          T (&out)[2]) {
  using P2 = typename ResPair<T>::type;
  res_apply<T, KR>(
      t, v, k, [&](int q) { return V[q]; },
      [&](int q, T(&o)[2]) {
        const P2 a = *reinterpret_cast<const P2 *>(V + q);
        o[0] = a.x;
        o[1] = a.y;
      },
      out);
}

// (A~ r~, r~) of the tile's cells; R holds r~ (synchronised).
template <typename T, int KR>
__device__ __forceinline__ double res_delta0(const ResTile<T, KR> &t, const T *R) {
  double d = 0.0;
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    T w[2];
    res_apply<T, KR>(t, t.r, R, k, w);
    d += (double)w[0] * (double)t.r[k][0];
    d += (double)w[1] * (double)t.r[k][1];
  }
  return d;
}

// The ring cells' outer neighbours as reduction c.tag published them (whole warps).
template <typename T, int KR>
__device__ __forceinline__ void res_ring_take(const ResCtx &c, ResTile<T, KR> &t) {
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const bool has = t.in[n] >= 0 || t.src[n];
    if (!__any_sync(0xffffffffu, has)) continue;
    const double v = res_wait(
        has,
        [&] {
          return t.src[n] ? res_ld(t.src[n] + (c.tag & 1) * res_edge(KR))
                          : res_lds(res_in_edge<KR>(c, c.tag, t.in[n]));
        },
        c.tag, c.sc, &c.sh->ok);
    if (has) t.r2[n] = T(v);
  }
}

// This thread's cell of the new residual R to the neighbour tile that reads it.
template <typename T, int KR>
__device__ __forceinline__ void res_publish(const ResCtx &c, const ResTile<T, KR> &t, const T *R) {
  if (t.qp < 0) return;
  const double v = R[t.qp];
  if (t.dst) res_st(t.dst + (c.tag & 1) * res_edge(KR), v, c.tag);
  else res_sts(c.tag & 1 ? t.out[1] : t.out[0], v, c.tag);
}

// A~ v of the ring cell (v1 its own value): cell(q) gives v at shared-memory position
// q, out[0 .. 2) its outer and diagonal neighbours'.
template <typename T, int KR, class C>
__device__ __forceinline__ T res_ring_apply(const ResTile<T, KR> &t, T v1, const T (&out)[2], C cell) {
  T v[4];
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    v[d] = cell(t.q1 + res_step(d));
    if ((t.dir & 3) == d) v[d] = out[0];
    if (t.dir >> 2 == d) v[d] = out[1];
  }
  const T off = res_off(t.h1[0], v[0], t.h1[1], v[1], t.h1[2], v[2], t.h1[3], v[3]);
  return t.dec >> 31 ? v1 : v1 - off;
}

// w = A~ r~ of the tile's cells (R synchronised) and this thread's part of
// (r~, r~), (w, r~), (p, w) and sum D r~^2 (diag(k): D = |Ct| of row k's cells).
template <int KR, class G>
__device__ __forceinline__ void res_stencil(const ResTile<double, KR> &t, const double *R, G diag,
                                            double (&w)[KR][2], double (&red)[kResSums]) {
  red[0] = red[1] = red[3] = red[5] = 0.0;
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    res_apply<double, KR>(t, t.r, R, k, w[k]);
    const double2 d = diag(k);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double uu = t.r[k][q] * t.r[k][q];
      red[0] += uu;
      red[1] += w[k][q] * t.r[k][q];
      red[3] += t.p[k][q] * w[k][q];
      red[5] += (q ? d.y : d.x) * uu;
    }
  }
}

// One FP32 sweep: p = r~ + beta p, r~ -= alpha A~ p, x += alpha p, and this thread's
// part of the five sums of sweep() in cg1.cu into red[0 .. 5).  A thread forms its
// neighbours' p from the shared copies P, R of the last sweep, so that one barrier
// separates the two stencils; Pn, Rn: this sweep's copies; p2: the directions of
// the ring cell's outer neighbours.
template <int KR>
__device__ __forceinline__ void res_sweep32(const ResCtx &c, ResTile<float, KR> &t, const float *P, const float *R,
                                            float *Pn, float *Rn, float alpha, float beta, float (&p2)[2],
                                            double (&red)[kResSums]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < kResSums; ++m) red[m] = 0.0;
  auto cell = [&](int q) -> float { return R[q] + beta * P[q]; };
  auto pair = [&](int q, float(&o)[2]) {
    const float2 a = *reinterpret_cast<const float2 *>(R + q), b = *reinterpret_cast<const float2 *>(P + q);
    o[0] = a.x + beta * b.x;
    o[1] = a.y + beta * b.y;
  };
#pragma unroll
  for (int k = 0; k < KR; ++k)
#pragma unroll
    for (int q = 0; q < 2; ++q) t.p[k][q] = t.r[k][q] + beta * t.p[k][q];
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    float s[2];
    res_apply<float, KR>(t, t.p, k, cell, pair, s);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      t.r[k][q] = t.r[k][q] - alpha * s[q];
      red[2] += (double)t.r[k][q] * (double)s[q];
      red[4] += (double)t.p[k][q] * (double)s[q];
    }
    const int at = res_q(2 * lane, wid * KR + k);
    *reinterpret_cast<float2 *>(Rn + at) = make_float2(t.r[k][0], t.r[k][1]);
    *reinterpret_cast<float2 *>(Pn + at) = make_float2(t.p[k][0], t.p[k][1]);
  }
  if (t.q1 >= 0) {
    const float p1 = t.r1 + beta * P[t.q1];
#pragma unroll
    for (int n = 0; n < 2; ++n) p2[n] = t.r2[n] + beta * p2[n];
    const float s = res_ring_apply<float, KR>(t, p1, p2, cell);
    t.r1 = t.r1 - alpha * s;
    Rn[t.q1] = t.r1;
    Pn[t.q1] = p1;
  }
  __syncthreads();
  res_publish<float, KR>(c, t, Rn);
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    float w[2];
    res_apply<float, KR>(t, t.r, Rn, k, w);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double u = t.r[k][q];
      red[0] += u * u;
      red[1] += (double)w[q] * u;
      red[3] += (double)t.p[k][q] * (double)w[q];
      t.x[k][q] = t.x[k][q] + alpha * t.p[k][q];
    }
  }
}

// What a mixed solve leaves: 0 after an error, 1 when done, 2 when the FP64 solve must
// take over, from the tag it ended with.
struct ResEnd {
  int code;
  unsigned tag;
};

// The CTA's place in the solve and the first tag: the domain's, or `from` if a solve of
// the same launch goes on from there (its other CTAs may not have read the domain's yet
// when this one leaves, so the two solves enter and leave once).  False after an error.
// sh and the dynamic shared memory belong to the caller's CTA.
__device__ __forceinline__ bool res_enter(const ResSys &s, unsigned rank, unsigned nb, unsigned csize, int KR,
                                          unsigned from, double *sm, ResShared *sh, ResCtx *c) {
  c->rank = rank;
  c->nb = nb;
  c->csize = csize;
  c->inbox = (unsigned)__cvta_generic_to_shared(sm + kResSums * kResThreads + 3 * res_arr(KR));
  c->sc = s.sc;
  c->sh = sh;
  c->sums = sm;
  c->slots = s.xbuf;
  c->edges = s.xbuf + 2L * nb * kResSlot + 2L * kResSlot * kResMaxGroups;
  __syncthreads();
  if (threadIdx.x == 0) {  // (a CTA that gave up may raise the tag meanwhile)
    sh->ok = 1;
    sh->beat = s.beat;
    sh->tag = from ? from : *(volatile unsigned *)&s.sc->res_tag;
  }
  __syncthreads();
  c->tag = sh->tag;
  if (from || c->tag < kResTagEnd) return true;
  // the tags near their end: every entry cleared, and the count starts again
  const long all = res_entries(nb, KR);
  for (long e = (long)rank * kResThreads + threadIdx.x; e < all; e += (long)nb * kResThreads)
    s.xbuf[e] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  if (nb > 1) {
    // a plain arrival count (all CTAs are co-resident), bounded like every wait
    if (threadIdx.x == 0) {
      const unsigned long long lim = s.sc->wait_limit_ns ? s.sc->wait_limit_ns : kBarrierTimeoutNs;
      const unsigned long long t0 = gtimer_ns();
      __threadfence();
      atomicAdd(&s.sc->bar_count, 1u);
      while (*(volatile unsigned *)&s.sc->bar_count < nb)
        if (gtimer_ns() - t0 > lim) {
          set_status(s.sc, FREHD_ERR_TIMEOUT);
          sh->ok = 0;
          break;
        }
      __threadfence();
    }
    __syncthreads();
    if (!sh->ok) return false;
  }
  c->tag = 0;
  return true;
}

// The solve's last act in each CTA.
__device__ __forceinline__ void res_leave(const ResSys &s, const ResCtx &c) {
  if (threadIdx.x != 0) return;
  if (*(volatile unsigned *)&s.sc->res_tag >= kResTagEnd && c.tag < kResTagEnd) {
    // after a restart of the tags (res_enter): every CTA has read the old one by now
    if (c.rank == 0) {
      s.sc->bar_count = 0;
      atomicExch(&s.sc->res_tag, c.tag);
    }
    return;
  }
  atomicMax(&s.sc->res_tag, c.tag);
}

// What a warp without a sum keeps of a sweep while the sums travel: the reciprocal of
// gamma = (r~, r~), scaled by a power of two where 1 / gamma would not be a normal
// number; in a batch also the sign of life.  (The division in the iteration's chain
// cost 2 us of a 59 us solve at 128 x 128 and 20 of 285 at 512 x 512.)
template <bool kBatch>
__device__ __forceinline__ void res_keep(const ResCtx &c, double gamma) {
  if (threadIdx.x >> 5 != kResSums) return;
  const double scale = gamma < 0x1p-512 ? 0x1p600 : gamma > 0x1p512 ? 0x1p-600 : 1.0;
  c.sh->scale = scale;
  c.sh->inv_gamma = 1.0 / (gamma * scale);
  if (kBatch && (c.tag & (kResBeat - 1)) == 0 && (threadIdx.x & 31) == 0) atomicAdd(c.sh->beat, 1u);
}

// beta = gamma / (the last sweep's gamma).
__device__ __forceinline__ double res_beta(double gamma, const ResShared *sh) {
  return gamma * sh->scale * sh->inv_gamma;
}

// FP64 solve by nb CTAs, of which this one is number `rank` = its tile number.
// sm: res_smem(KR) bytes of shared memory.  from: see res_enter.  kBatch: other solves
// wait for this one's signs of life (s.beat).  False after an error
// (status set).
template <int KR, bool kBatch>
__device__ __forceinline__ bool res_fp64(const ResSys &s, unsigned rank, unsigned nb, unsigned csize, unsigned from,
                                         double *sm, ResShared *sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx);
  const int i0 = (int)(rank % ntx) * kResTW, j0 = (int)(rank / ntx) * res_th(KR);
  double *R = sm + kResSums * kResThreads;
  ResCtx c;
  if (!res_enter(s, rank, nb, csize, KR, from, sm, sh, &c)) return false;
  ResTile<double, KR> t;
  double w[KR][2], as[KR][2];  // A~ r~, A~ p
  // x~ and |Ct| of the tallest tile's cells lie in shared memory, those of the others in
  // registers.  128 a thread do not hold all of it even so: 708 bytes of spill loads a
  // thread for the tallest tile, 308 with two rows and 88 with one, partly in the set-up
  constexpr bool kShared = KR == kResMaxKR;
  double D[kShared ? 1 : KR][2];
  double2 *const xs = reinterpret_cast<double2 *>(R + res_arr(KR)) + threadIdx.x, *const Ds = xs + KR * kResThreads;
  static_assert(4 * KR * kResThreads <= 2 * res_arr(KR), "both fit the set-up's arrays");
  int it = 0, it_all = 0, fallback = 0;
  double rr = 0.0, bnorm = 0.0, limit = 0.0;
  bool ok = true;
  for (int attempt = 0;; ++attempt) {
    const int elim = s.eliminate | (attempt > 0);
    res_setup<double, KR>(s, c, i0, j0, elim, R, t);
    double red[kResSums] = {0, 0, 0, 0, 0, 0};
    if (s.x0 || elim) {
      const double *x0 = s.x0;
      res_start<double, KR>(s, i0, j0, R, t, red, [&](int i, int j) {
        return res_residual(s, i, j, elim, [&](long k) { return x0 ? x0[k] : 0.0; });
      });
    } else {
      res_start<double, KR>(s, i0, j0, R, t, red,
                            [&](int i, int j) { return s.b[s.off + (long)j * s.pitch + i]; });
    }
    // (every thread has read its couplings: res_start synchronised)
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      double d[2], x[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
        d[q] = x[q] = as[k][q] = 0.0;
        if (res_in(s, i, j)) {
          const long kk = s.off + (long)j * s.pitch + i;
          d[q] = fabs(s.Ct[kk]);
          if (s.x0) x[q] = sqrt(d[q]) * s.x0[kk];
        }
        if (!kShared) {
          D[kShared ? 0 : k][q] = d[q];
          t.x[k][q] = x[q];
        }
      }
      if (kShared) {
        Ds[k * kResThreads] = make_double2(d[0], d[1]);
        xs[k * kResThreads] = make_double2(x[0], x[1]);
      }
    }
    auto diag = [&](int k) {
      return kShared ? Ds[k * kResThreads] : make_double2(D[kShared ? 0 : k][0], D[kShared ? 0 : k][1]);
    };
    const double bb = red[2];
    double first[kResSums], rr0 = red[1], s1 = 0.0, w1 = 0.0;
    res_stencil<KR>(t, R, diag, w, first);
    auto ring_stencil = [&] {
      if (t.q1 >= 0) w1 = res_ring_apply<double, KR>(t, t.r1, t.r2, [&](int q) { return R[q]; });
    };
    ring_stencil();
    red[0] = first[0];
    red[1] = rr0;
    red[2] = bb;
    red[3] = first[1];
    ++c.tag;
    if (!(ok = res_allreduce<4>(red, c, [] {}))) break;
    double gamma = red[0], delta = red[3], e1 = 0.0, e2 = 0.0, e3 = 0.0;
    rr = red[1];
    bnorm = sqrt(red[2]);
    limit = res_limit(bnorm, s.eps);
    double best = rr;
    int best_it = 0;
    bool stalled = false;
    it = 0;
    while (!(rr <= limit) && it < s.max_iter) {
      const double beta = it == 0 ? 0.0 : res_beta(gamma, sh);
      const double alpha = gamma / (delta + beta * (e1 + e2) + beta * beta * e3);
      ++it;
      ++c.tag;
      red[2] = red[4] = 0.0;
#pragma unroll
      for (int k = 0; k < KR; ++k) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          t.p[k][q] = t.r[k][q] + beta * t.p[k][q];
          as[k][q] = w[k][q] + beta * as[k][q];
          t.r[k][q] = t.r[k][q] - alpha * as[k][q];
        }
        *reinterpret_cast<double2 *>(R + res_q(2 * lane, wid * KR + k)) = make_double2(t.r[k][0], t.r[k][1]);
      }
      if (t.q1 >= 0) {
        s1 = w1 + beta * s1;
        t.r1 = t.r1 - alpha * s1;
        R[t.q1] = t.r1;
      }
      __syncthreads();
      res_publish<double, KR>(c, t, R);
      res_stencil<KR>(t, R, diag, w, red);
#pragma unroll
      for (int k = 0; k < KR; ++k) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          red[2] += t.r[k][q] * as[k][q];
          red[4] += t.p[k][q] * as[k][q];
          if (!kShared) t.x[k][q] = t.x[k][q] + alpha * t.p[k][q];
        }
        if (kShared) {
          double2 x = xs[k * kResThreads];
          x.x += alpha * t.p[k][0];
          x.y += alpha * t.p[k][1];
          xs[k * kResThreads] = x;
        }
      }
      ok = res_allreduce<6>(red, c, [&] {
        res_keep<kBatch>(c, gamma);
        res_ring_take<double, KR>(c, t);
        ring_stencil();
      });
      if (!ok) break;
      gamma = red[0];
      delta = red[1];
      e1 = red[2];
      e2 = red[3];
      e3 = red[4];
      rr = red[5];
      if (rr < 0.25 * best) {
        best = rr;
        best_it = it;
      } else if (!elim && it - best_it >= kStallIters) {
        stalled = true;
        break;
      }
    }
    if (!ok) break;
    it_all += it;
    if (!stalled) break;
    fallback = 1;
  }
  if (ok) {
    // x = x~/sqrt|Ct|, by way of the shared array (R is free: the last reduction ended)
#pragma unroll
    for (int k = 0; k < KR; ++k)
      *reinterpret_cast<double2 *>(R + res_q(2 * lane, wid * KR + k)) =
          kShared ? xs[k * kResThreads] : make_double2(t.x[k][0], t.x[k][1]);
    __syncthreads();
#pragma unroll 1
    for (int e = threadIdx.x; e < kResTW * res_th(KR); e += kResThreads) {
      const int lx = e % kResTW, ly = e / kResTW, i = i0 + lx, j = j0 + ly;
      if (res_in(s, i, j)) {
        const long k = s.off + (long)j * s.pitch + i;
        // (a start that meets the tolerance is the solution, to the last bit)
        s.x[k] = it_all > 0 ? R[res_q(lx, ly)] / sqrt(fabs(s.Ct[k])) : s.x0 ? s.x0[k] : 0.0;
      }
    }
    if (rank == 0 && threadIdx.x == 0) {
      s.sc->cg_iters = it_all;
      s.sc->cg_fallback = fallback;
      s.sc->cg_noconv = !(rr <= limit);
      s.sc->cg_rr = rr;
      s.sc->cg_bb = bnorm * bnorm;
    }
  }
  res_leave(s, c);
  return ok;
}

// Mixed-precision solve: FP32 inner solves on the resident tile inside FP64
// refinement (cg1_mixed in cg1.cu, same steps, same stopping rules).  x lives in
// registers; between two inner solves it goes through global memory, where the
// next residual reads its neighbours.
template <int KR, bool kBatch>
__device__ __forceinline__ ResEnd res_mixed(const ResSys &s, double eps_inner, unsigned rank, unsigned nb, unsigned csize,
                                         double *sm, ResShared *sh) {
  constexpr int kArr = res_arr(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx);
  const int i0 = (int)(rank % ntx) * kResTW, j0 = (int)(rank / ntx) * res_th(KR);
  double *ds = sm + kResSums * kResThreads;
  float *P = reinterpret_cast<float *>(ds), *R = P + kArr;  // the other copies lie 2 kArr further
  ResCtx c;
  if (!res_enter(s, rank, nb, csize, KR, 0, sm, sh, &c)) return ResEnd{0, 0};
  ResTile<float, KR> t;
  double xd[KR][2];
#pragma unroll
  for (int k = 0; k < KR; ++k)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
      xd[k][q] = s.x0 && res_in(s, i, j) ? s.x0[s.off + (long)j * s.pitch + i] : 0.0;
    }
  res_setup<float, KR>(s, c, i0, j0, s.eliminate, ds, t);
  double rr = 0.0, rr_prev = 0.0, bnorm = 0.0, limit = 0.0;
  int it_all = 0, ret = 2;
  for (int outer = 0; outer < kResMaxOuter; ++outer) {
    // r = b - A x in FP64, r~ = r/sqrt|Ct| in FP32
    double red[kResSums] = {0, 0, 0, 0, 0, 0};
    if (outer == 0) {
      const double *x0 = s.x0;
      if (x0 || s.eliminate)
        res_start<float, KR>(s, i0, j0, R, t, red, [&](int i, int j) {
          return res_residual(s, i, j, s.eliminate, [&](long k) { return x0 ? x0[k] : 0.0; });
        });
      else
        res_start<float, KR>(s, i0, j0, R, t, red,
                             [&](int i, int j) { return s.b[s.off + (long)j * s.pitch + i]; });
    } else {
      const double *x = s.x;
      res_start<float, KR>(s, i0, j0, R, t, red,
                           [&](int i, int j) { return res_residual_padded(s, x, i, j, s.eliminate); });
    }
    // p = 0 on the tile and its ring (read only after the reduction's barriers)
#pragma unroll
    for (int k = 0; k < KR; ++k)
      *reinterpret_cast<float2 *>(P + res_q(2 * lane, wid * KR + k)) = make_float2(0.0f, 0.0f);
    if (t.q1 >= 0) P[t.q1] = 0.0f;
    float p2[2] = {0.0f, 0.0f};
    red[3] = res_delta0<float, KR>(t, R);
    ++c.tag;
    if (!res_allreduce<4>(red, c, [] {})) {
      ret = 0;
      break;
    }
    rr = red[1];
    if (outer == 0) {
      bnorm = sqrt(red[2]);
      limit = res_limit(bnorm, s.eps);
    }
    if (rr <= limit) {
      ret = 1;
      break;
    }
    if (outer > 0 && rr > 1e-2 * rr_prev) break;  // no tenfold gain: FP64 takes over
    rr_prev = rr;
    // A~ d~ = r~ until (r~, r~) fell by eps_inner^2
    double gamma = red[0], delta = red[3], e1 = 0.0, e2 = 0.0, e3 = 0.0;
    const double stop = eps_inner * eps_inner * gamma;
#pragma unroll
    for (int k = 0; k < KR; ++k) t.x[k][0] = t.x[k][1] = 0.0f;
    int it = 0;
    bool ok = true;
    while (gamma > stop && it < s.max_iter) {
      const double beta = it == 0 ? 0.0 : res_beta(gamma, sh);
      const double alpha = gamma / (delta + beta * (e1 + e2) + beta * beta * e3);
      const int cur = it & 1;
      ++it;
      ++c.tag;
      res_sweep32<KR>(c, t, P + 2 * cur * kArr, R + 2 * cur * kArr, P + 2 * (cur ^ 1) * kArr,
                      R + 2 * (cur ^ 1) * kArr, (float)alpha, (float)beta, p2, red);
      ok = res_allreduce<5>(red, c, [&] {
        res_keep<kBatch>(c, gamma);
        res_ring_take<float, KR>(c, t);
      });
      if (!ok) break;
      gamma = red[0];
      delta = red[1];
      e1 = red[2];
      e2 = red[3];
      e3 = red[4];
    }
    if (!ok) {
      ret = 0;
      break;
    }
    it_all += it;
    // x += d~/sqrt|Ct| (the correction needs FP32 accuracy only: the next residual is
    // exact in FP64 for whatever x results)
#pragma unroll
    for (int k = 0; k < KR; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
        if (res_in(s, i, j)) {
          const long kk = s.off + (long)j * s.pitch + i;
          const float fs = (float)(1.0 / sqrt(fabs(s.Ct[kk])));
          if (it > 0) xd[k][q] = fma((double)t.x[k][q], (double)fs, xd[k][q]);
          s.x[kk] = xd[k][q];
        }
      }
    // (x by this CTA's threads, before the block barrier; the neighbours' after it)
    ++c.tag;
    if (!res_allreduce<1, true>(red, c, [] {})) {
      ret = 0;
      break;
    }
  }
  if (ret == 1) {
    if (it_all == 0) {  // converged at the start: x was never stored
#pragma unroll
      for (int k = 0; k < KR; ++k)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
          if (res_in(s, i, j)) s.x[s.off + (long)j * s.pitch + i] = xd[k][q];
        }
    }
    if (rank == 0 && threadIdx.x == 0) {
      s.sc->cg_iters = it_all;
      s.sc->cg_fallback = 0;
      s.sc->cg_noconv = 0;
      s.sc->cg_rr = rr;
      s.sc->cg_bb = bnorm * bnorm;
    }
  }
  if (ret != 2) res_leave(s, c);
  return ResEnd{ret, c.tag};
}

}  // namespace

}  // namespace frehd

#endif
