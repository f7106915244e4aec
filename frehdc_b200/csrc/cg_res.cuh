// Resident Jacobi-PCG: the single-sweep solve of cg1.cu (same scaled system,
// same recurrences, same stopping rule and fall-back) for domains whose solver
// state fits on chip.
//
// What bounds a small solve is not traffic but the latency of an iteration: with
// the state in HBM every iteration waits for its TMA boxes and for a two-hop
// grid reduction (arrive, last block sums and publishes, everyone reads), 11 us
// per iteration at 128 x 128.  Here each CTA keeps one tile of
// 64 x (16 KR) cells for the whole solve: residual, direction, solution and
// couplings in registers, with copies of the residual and the direction in shared
// memory where the stencil's neighbours read them.  An iteration then touches
// global memory twice, both in one hop:
//   * the tile's outer second row and column of the new residual (what a
//     neighbour tile cannot compute itself: it recomputes the first ring), and
//   * the CTA's six partial sums, which every CTA reads from every other and adds
//     in rank order (the same total everywhere, in a fixed order).
// Both travel as 16-byte entries {low word, tag, high word, tag}: the tag is the
// reduction's number, so an entry announces itself and neither a fence nor an
// arrival counter stands between the writer's store and the reader's load.  The
// entries alternate between two buffers by tag parity; no CTA can write the
// buffer of reduction t + 2 before every CTA has published t + 1, that is,
// finished reading t.
//
// Tags only grow: a launch starts at Scratch::res_tag, and every CTA raises it
// to the last tag it used, whether it ends well or after a wait that gave up.
#ifndef FREHD_CG_RES_CUH
#define FREHD_CG_RES_CUH

#include "cg_common.cuh"
#include "cg_res.h"

namespace frehd {

// The system of one solve.  Cell (i, j) at off + j * pitch + i of every array;
// nothing outside 0 <= i < nx, 0 <= j < ny is read.
struct ResSys {
  int nx, ny;
  long pitch, off;
  const double *Ct, *Gx, *Gy, *b, *x0;  // x0 null: the solve starts from zero
  double *x;
  double eps;
  int max_iter, eliminate;
  Scratch *sc;
  uint4 *xbuf;
};

struct ResShared {
  double part[NWARP][kResSlot], part2[NWARP][kResSlot];
  int ok;
};

// Where a CTA stands: its rank among the nb of the solve, the tag of the last
// reduction, and the buffers.
struct ResCtx {
  unsigned rank, nb, tag;
  uint4 *slots, *edges;
  Scratch *sc;
  ResShared *sh;
};

namespace {

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

// The entry's value once it carries `tag`; the wait is bounded (ok becomes 0).
__device__ __forceinline__ double res_wait(const uint4 *a, unsigned tag, Scratch *sc, int *ok) {
  uint4 v = res_ld(a);
  if (v.y == tag && v.w == tag) return res_val(v);
  const unsigned long long lim = sc->wait_limit_ns ? sc->wait_limit_ns : kBarrierTimeoutNs;
  const unsigned long long t0 = gtimer_ns();
  for (unsigned n = 1;; ++n) {
    v = res_ld(a);
    if (v.y == tag && v.w == tag) return res_val(v);
    if ((n & 63u) == 0) {
      if (*(volatile int *)&sc->status == FREHD_ERR_TIMEOUT || gtimer_ns() - t0 > lim) {
        set_status(sc, FREHD_ERR_TIMEOUT);
        *(volatile int *)ok = 0;
        return 0.0;
      }
    }
  }
}

// Sum of eight values over a warp: three halving exchanges leave each lane one
// of them (number res_lane_sum(lane)), two more add the rest.
__device__ __forceinline__ int res_lane_sum(int lane) {
  return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}
__device__ __forceinline__ double res_warp_sums(const double (&v)[8], int lane) {
  double a[4], b[2];
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    a[q] = (h4 ? v[q + 4] : v[q]) + __shfl_xor_sync(0xffffffffu, h4 ? v[q] : v[q + 4], 16);
#pragma unroll
  for (int q = 0; q < 2; ++q)
    b[q] = (h3 ? a[q + 2] : a[q]) + __shfl_xor_sync(0xffffffffu, h3 ? a[q] : a[q + 2], 8);
  double c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}
// Lane l: the total of value l & 7 over the warps' entries.
__device__ __forceinline__ double res_gather(const double (*s)[kResSlot], int lane) {
  const int m = lane & 7, w = (lane >> 3) * (NWARP / 4);
  double t = s[w][m];
#pragma unroll
  for (int q = 1; q < NWARP / 4; ++q) t += s[w + q][m];
  t += __shfl_xor_sync(0xffffffffu, t, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 16);
  return t;
}

// v[0 .. NV) summed over all threads of the solve's CTAs, the same in each, and a
// barrier among them (for the entries stored before it under this tag).
// ++tag is the caller's.
template <int NV>
__device__ __forceinline__ bool res_allreduce(double (&v)[8], const ResCtx &c) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  ResShared *sh = c.sh;
  const double mine = res_warp_sums(v, lane);
  if (!(lane & 3)) sh->part[wid][res_lane_sum(lane)] = mine;
  __syncthreads();
  double t;
  if (c.nb == 1) {
    t = res_gather(sh->part, lane);
  } else {
    uint4 *sl = c.slots + (long)(c.tag & 1) * c.nb * kResSlot;
    if (wid == 0) {
      t = res_gather(sh->part, lane);
      if (lane < NV) res_st(sl + (long)c.rank * kResSlot + lane, t, c.tag);
    }
    // every CTA's sums in rank order: thread (warp, lane) takes value lane & 7 of
    // ranks 4 warp + lane / 8, + 64, ...
    double acc = 0.0;
    if ((lane & 7) < NV)
      for (unsigned s = 4 * wid + (lane >> 3); s < c.nb; s += 4 * NWARP)
        acc += res_wait(sl + (long)s * kResSlot + (lane & 7), c.tag, c.sc, &sh->ok);
    __syncwarp();
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    if (lane < 8) sh->part2[wid][lane] = acc;
    __syncthreads();
    if (!*(volatile int *)&sh->ok) return false;
    t = res_gather(sh->part2, lane);
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = __shfl_sync(0xffffffffu, t, q);
  return true;
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

// A thread's part of the tile: KR rows of two cells, and at most one cell each
// of the first and of the second ring around the tile.
template <typename T, int KR>
struct ResTile {
  T r[KR][2], p[KR][2], x[KR][2];
  T hx[KR][3], hy[KR + 1][2];  // |couplings| of the rows' x faces (west, middle, east) and y faces
  T r1, p1, h1[4], r2, p2;     // h1: east, west, north, south
  unsigned dec;                // bit 2k + c: decoupled cell; bit 31: decoupled ring cell
  int q1, q2;                  // shared-memory positions of the ring cells (-1: none)
  const uint4 *src;            // exchange entry (parity 0) of the second-ring cell, or null
};

// Tile coordinates of ring cells: number e of the first ring (2 TW + 2 TH of
// them) and of the second (those at distance two straight, and the four diagonal ones).
template <int KR>
__device__ __forceinline__ bool res_ring1(int e, int *lx, int *ly) {
  constexpr int TH = res_th(KR);
  if (e < kResTW) { *lx = e; *ly = -1; return true; }
  e -= kResTW;
  if (e < kResTW) { *lx = e; *ly = TH; return true; }
  e -= kResTW;
  if (e < TH) { *lx = -1; *ly = e; return true; }
  e -= TH;
  *lx = kResTW; *ly = e;
  return e < TH;
}

// The second-ring cell's place and, in the neighbour tile (dx, dy), the exchange
// entry that holds it: west column | east column | south row | north row |
// corners south-west, south-east, north-west, north-east.
template <int KR>
__device__ __forceinline__ bool res_ring2(int e, int *lx, int *ly, int *dx, int *dy, int *entry) {
  constexpr int TH = res_th(KR), TW = kResTW;
  *dx = *dy = 0;
  if (e < TW) { *lx = e; *ly = -2; *dy = -1; *entry = 2 * TH + TW + e; return true; }
  e -= TW;
  if (e < TW) { *lx = e; *ly = TH + 1; *dy = 1; *entry = 2 * TH + e; return true; }
  e -= TW;
  if (e < TH) { *lx = -2; *ly = e; *dx = -1; *entry = TH + e; return true; }
  e -= TH;
  if (e < TH) { *lx = TW + 1; *ly = e; *dx = 1; *entry = e; return true; }
  e -= TH;
  if (e >= 4) return false;
  // my south-west diagonal cell is that tile's north-east corner, and so on
  *dx = (e & 1) ? 1 : -1;
  *dy = (e & 2) ? 1 : -1;
  *lx = (e & 1) ? TW : -1;
  *ly = (e & 2) ? TH : -1;
  *entry = 2 * TH + 2 * TW + (3 - e);
  return true;
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

// The tile's couplings (scaled, |.|), decoupled flags and ring bookkeeping.  sm:
// the CTA's shared memory, used for sqrt|Ct| (negative on decoupled rows) of
// the tile and its two rings; on return it is free again.
template <typename T, int KR>
__device__ __forceinline__ void res_setup(const ResSys &s, const ResCtx &c, int i0, int j0, int elim,
                                          double *ds, ResTile<T, KR> &t) {
  constexpr int TH = res_th(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx), nty = (s.ny + TH - 1) / TH;
  __syncthreads();
  for (int e = threadIdx.x; e < (TH + 4) * kResPitch; e += kCgThreads) {
    const int i = i0 + e % kResPitch - 2, j = j0 + e / kResPitch - 2;
    double d = -1.0;
    if (res_in(s, i, j)) {
      const double ct = s.Ct[s.off + (long)j * s.pitch + i];
      d = ct < 0 ? -sqrt(-ct) : sqrt(ct);
    }
    ds[e] = d;
  }
  __syncthreads();
  // coupling across the east (dy = 0) or north face of tile cell (lx, ly)
  auto face = [&](int lx, int ly, int dx, int dy) -> T {
    const int i = i0 + lx, j = j0 + ly;
    if (!res_in(s, i, j) || !res_in(s, i + dx, j + dy)) return T(0);
    const double a = ds[res_q(lx, ly)], b = ds[res_q(lx + dx, ly + dy)];
    if (elim && !(a > 0 && b > 0)) return T(0);
    const double g = (dx ? s.Gx : s.Gy)[s.off + (long)j * s.pitch + i];
    const double h = g / (fabs(a) * fabs(b));
    return dx ? T(fabs(T(h))) : T(h);
  };
  t.dec = 0;
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int ly = wid * KR + k, lx = 2 * lane;
    t.hx[k][0] = face(lx - 1, ly, 1, 0);
    t.hx[k][1] = face(lx, ly, 1, 0);
    t.hx[k][2] = face(lx + 1, ly, 1, 0);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (k == 0) t.hy[0][q] = face(lx + q, ly - 1, 0, 1);
      t.hy[k + 1][q] = face(lx + q, ly, 0, 1);
      if (ds[res_q(lx + q, ly)] < 0) t.dec |= 1u << (2 * k + q);
    }
  }
  t.q1 = t.q2 = -1;
  t.src = nullptr;
  t.r1 = t.p1 = t.r2 = t.p2 = T(0);
#pragma unroll
  for (int q = 0; q < 4; ++q) t.h1[q] = T(0);
  int lx, ly;
  if (res_ring1<KR>(threadIdx.x, &lx, &ly)) {
    t.q1 = res_q(lx, ly);
    t.h1[0] = face(lx, ly, 1, 0);
    t.h1[1] = face(lx - 1, ly, 1, 0);
    t.h1[2] = face(lx, ly, 0, 1);
    t.h1[3] = face(lx, ly - 1, 0, 1);
    if (ds[t.q1] < 0) t.dec |= 1u << 31;
  }
  int dx, dy, entry;
  if (res_ring2<KR>(kCgThreads - 1 - (int)threadIdx.x, &lx, &ly, &dx, &dy, &entry)) {
    t.q2 = res_q(lx, ly);
    const int bx = (int)(c.rank % ntx) + dx, by = (int)(c.rank / ntx) + dy;
    if ((unsigned)bx < (unsigned)ntx && (unsigned)by < (unsigned)nty)
      t.src = c.edges + ((long)by * ntx + bx) * 2 * res_edge(KR) + entry;
  }
  __syncthreads();
}

// r~ (of a residual function of the interior cells) into the tile and its rings
// and shared memory; adds (r~, r~) and ||r||^2 to acc[0], acc[1] and ||b||^2 to acc[2].
template <typename T, int KR, class F>
__device__ __forceinline__ void res_start(const ResSys &s, int i0, int j0, T *R, ResTile<T, KR> &t,
                                          double (&acc)[8], F resid) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto scaled = [&](int i, int j, double *r) -> T {
    if (!res_in(s, i, j)) return T(0);
    *r = resid(i, j);
    return T(*r / sqrt(fabs(s.Ct[s.off + (long)j * s.pitch + i])));
  };
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int ly = wid * KR + k;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + 2 * lane + q, j = j0 + ly;
      double r = 0.0;
      const T rs = scaled(i, j, &r);
      t.r[k][q] = rs;
      t.p[k][q] = T(0);
      R[res_q(2 * lane + q, ly)] = rs;
      acc[0] += (double)rs * (double)rs;
      acc[1] += r * r;
      if (res_in(s, i, j)) {
        const double bk = s.b[s.off + (long)j * s.pitch + i];
        acc[2] += bk * bk;
      }
    }
  }
  double unused;
  if (t.q1 >= 0) {
    t.r1 = scaled(i0 + t.q1 % kResPitch - 2, j0 + t.q1 / kResPitch - 2, &unused);
    t.p1 = T(0);
    R[t.q1] = t.r1;
  }
  if (t.q2 >= 0) {
    t.r2 = scaled(i0 + t.q2 % kResPitch - 2, j0 + t.q2 / kResPitch - 2, &unused);
    t.p2 = T(0);
  }
}

// A~ v of a thread's cells (row k): v its own values, V the array in shared memory.
template <typename T, int KR>
__device__ __forceinline__ void res_apply(const ResTile<T, KR> &t, const T (&v)[KR][2], const T *V, int k,
                                          T (&out)[2]) {
  using P2 = typename ResPair<T>::type;
  const int lane = threadIdx.x & 31, ly = (threadIdx.x >> 5) * KR + k;
  const int q = res_q(2 * lane, ly);
  T south[2], north[2];
  if (k == 0) {
    const P2 a = *reinterpret_cast<const P2 *>(V + q - kResPitch);
    south[0] = a.x;
    south[1] = a.y;
  } else {
    south[0] = v[k > 0 ? k - 1 : 0][0];
    south[1] = v[k > 0 ? k - 1 : 0][1];
  }
  if (k == KR - 1) {
    const P2 a = *reinterpret_cast<const P2 *>(V + q + kResPitch);
    north[0] = a.x;
    north[1] = a.y;
  } else {
    north[0] = v[k < KR - 1 ? k + 1 : k][0];
    north[1] = v[k < KR - 1 ? k + 1 : k][1];
  }
  T west = __shfl_up_sync(0xffffffffu, v[k][1], 1), east = __shfl_down_sync(0xffffffffu, v[k][0], 1);
  if (lane == 0) west = V[q - 1];
  if (lane == 31) east = V[q + 2];
  const T off0 = t.hx[k][1] * v[k][1] + t.hx[k][0] * west + t.hy[k + 1][0] * north[0] + t.hy[k][0] * south[0];
  const T off1 = t.hx[k][2] * east + t.hx[k][1] * v[k][0] + t.hy[k + 1][1] * north[1] + t.hy[k][1] * south[1];
  out[0] = (t.dec >> (2 * k)) & 1u ? v[k][0] : v[k][0] - off0;
  out[1] = (t.dec >> (2 * k + 1)) & 1u ? v[k][1] : v[k][1] - off1;
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

// One sweep: p = r~ + beta p, r~ -= alpha A~ p, x += alpha p, and this thread's
// part of the six sums of sweep() in cg1.cu into red[0 .. 6).  first: the rings'
// residuals are still those of res_start.  D: |Ct| of the cells (kUnscaled).
template <typename T, int KR, bool kUnscaled>
__device__ __forceinline__ void res_sweep(const ResCtx &c, ResTile<T, KR> &t, T *P, T *R, T alpha, T beta,
                                          bool first, const double (&D)[KR][2], int bx, int by, int ntx,
                                          int nty, double (&red)[8]) {
  using P2 = typename ResPair<T>::type;
  constexpr int TH = res_th(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < 8; ++m) red[m] = 0.0;
  // p on the tile and both rings
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    t.p[k][0] = t.r[k][0] + beta * t.p[k][0];
    t.p[k][1] = t.r[k][1] + beta * t.p[k][1];
    P2 a;
    a.x = t.p[k][0];
    a.y = t.p[k][1];
    *reinterpret_cast<P2 *>(P + res_q(2 * lane, wid * KR + k)) = a;
  }
  if (t.q1 >= 0) {
    t.p1 = t.r1 + beta * t.p1;
    P[t.q1] = t.p1;
  }
  if (t.q2 >= 0) {
    if (!first && t.src)  // published under the previous reduction's tag
      t.r2 = T(res_wait(t.src + ((c.tag - 1) & 1) * res_edge(KR), c.tag - 1, c.sc, &c.sh->ok));
    t.p2 = t.r2 + beta * t.p2;
    P[t.q2] = t.p2;
  }
  __syncthreads();
  // r~ on the tile and the first ring; the outer second row and column go out
  uint4 *mine = c.edges + ((long)by * ntx + bx) * 2 * res_edge(KR) + (c.tag & 1) * res_edge(KR);
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    T s[2];
    res_apply<T, KR>(t, t.p, P, k, s);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      t.r[k][q] = t.r[k][q] - alpha * s[q];
      red[2] += (double)t.r[k][q] * (double)s[q];
      red[4] += (double)t.p[k][q] * (double)s[q];
    }
    const int ly = wid * KR + k;
    P2 a;
    a.x = t.r[k][0];
    a.y = t.r[k][1];
    *reinterpret_cast<P2 *>(R + res_q(2 * lane, ly)) = a;
    if (c.nb > 1) {
      if (ly == 1 && by > 0) {
        res_st(mine + 2 * TH + 2 * lane, (double)t.r[k][0], c.tag);
        res_st(mine + 2 * TH + 2 * lane + 1, (double)t.r[k][1], c.tag);
      }
      if (ly == TH - 2 && by + 1 < nty) {
        res_st(mine + 2 * TH + kResTW + 2 * lane, (double)t.r[k][0], c.tag);
        res_st(mine + 2 * TH + kResTW + 2 * lane + 1, (double)t.r[k][1], c.tag);
      }
      if (lane == 0 && bx > 0) {
        res_st(mine + ly, (double)t.r[k][1], c.tag);
        if (ly == 0 || ly == TH - 1)
          res_st(mine + 2 * TH + 2 * kResTW + (ly ? 2 : 0), (double)t.r[k][0], c.tag);
      }
      if (lane == 31 && bx + 1 < ntx) {
        res_st(mine + TH + ly, (double)t.r[k][0], c.tag);
        if (ly == 0 || ly == TH - 1)
          res_st(mine + 2 * TH + 2 * kResTW + (ly ? 3 : 1), (double)t.r[k][1], c.tag);
      }
    }
  }
  if (t.q1 >= 0) {
    const T off = t.h1[0] * P[t.q1 + 1] + t.h1[1] * P[t.q1 - 1] + t.h1[2] * P[t.q1 + kResPitch] +
                  t.h1[3] * P[t.q1 - kResPitch];
    const T s = (t.dec >> 31) ? t.p1 : t.p1 - off;
    t.r1 = t.r1 - alpha * s;
    R[t.q1] = t.r1;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    T w[2];
    res_apply<T, KR>(t, t.r, R, k, w);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double u = t.r[k][q];
      red[0] += u * u;
      red[1] += (double)w[q] * u;
      red[3] += (double)t.p[k][q] * (double)w[q];
      if (kUnscaled) red[5] += D[k][q] * (u * u);
      t.x[k][q] = t.x[k][q] + alpha * t.p[k][q];
    }
  }
}

__device__ __forceinline__ bool res_converged(double rr, double bnorm, double eps) {
  const double rn = sqrt(rr);
  return rn < eps * bnorm || (bnorm == 0.0 && 1.0 + rn == 1.0);
}

// The CTA's place in the solve and the first tag; false after an error.  sh and
// the dynamic shared memory belong to the caller's CTA.
__device__ __forceinline__ bool res_enter(const ResSys &s, unsigned rank, unsigned nb, int KR, ResShared *sh,
                                          ResCtx *c) {
  c->rank = rank;
  c->nb = nb;
  c->sc = s.sc;
  c->sh = sh;
  c->slots = s.xbuf;
  c->edges = s.xbuf + 2L * nb * kResSlot;
  __syncthreads();
  if (threadIdx.x == 0) sh->ok = 1;
  c->tag = *(volatile unsigned *)&s.sc->res_tag;
  if (c->tag < 0xC0000000u) return true;
  // the tags near their end: every entry cleared, and the count starts again
  const long per = 2L * (kResSlot + res_edge(KR));
  for (long e = threadIdx.x; e < per; e += kCgThreads)
    s.xbuf[(long)rank * per + e] = make_uint4(0, 0, 0, 0);
  __threadfence();
  __syncthreads();
  if (nb > 1) {
    // a plain arrival count (all CTAs are co-resident), bounded like every wait
    if (threadIdx.x == 0) {
      const unsigned long long t0 = gtimer_ns();
      atomicAdd(&s.sc->bar_count, 1u);
      while (*(volatile unsigned *)&s.sc->bar_count < nb)
        if (gtimer_ns() - t0 > kBarrierTimeoutNs) {
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
  if (*(volatile unsigned *)&s.sc->res_tag >= 0xC0000000u && c.tag < 0x40000000u) {
    // after a restart of the tags (res_enter): every CTA has read the old one by now
    if (c.rank == 0) {
      s.sc->bar_count = 0;
      atomicExch(&s.sc->res_tag, c.tag);
    }
    return;
  }
  atomicMax(&s.sc->res_tag, c.tag);
}

// FP64 solve by nb CTAs, of which this one is number `rank` = its tile number.
// sm: res_smem(KR) bytes of shared memory.  False after an error (status set).
template <int KR>
__device__ __forceinline__ bool res_fp64(const ResSys &s, unsigned rank, unsigned nb, double *sm, ResShared *sh) {
  constexpr int TH = res_th(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx), nty = (s.ny + TH - 1) / TH;
  const int bx = (int)(rank % ntx), by = (int)(rank / ntx);
  const int i0 = bx * kResTW, j0 = by * TH;
  double *P = sm, *R = sm + (TH + 4) * kResPitch;
  ResCtx c;
  if (!res_enter(s, rank, nb, KR, sh, &c)) return false;
  ResTile<double, KR> t;
  double D[KR][2];
  int it = 0, it_all = 0, fallback = 0, noconv = 0;
  double rr = 0.0, bnorm = 0.0;
  bool ok = true;
  for (int attempt = 0;; ++attempt) {
    const int elim = s.eliminate | (attempt > 0);
    res_setup<double, KR>(s, c, i0, j0, elim, sm, t);
    double red[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (s.x0 || elim) {
      const double *x0 = s.x0;
      res_start<double, KR>(s, i0, j0, R, t, red, [&](int i, int j) {
        return res_residual(s, i, j, elim, [&](long k) { return x0 ? x0[k] : 0.0; });
      });
    } else {
      res_start<double, KR>(s, i0, j0, R, t, red,
                            [&](int i, int j) { return s.b[s.off + (long)j * s.pitch + i]; });
    }
#pragma unroll
    for (int k = 0; k < KR; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
        D[k][q] = 0.0;
        t.x[k][q] = 0.0;
        if (res_in(s, i, j)) {
          const long kk = s.off + (long)j * s.pitch + i;
          D[k][q] = fabs(s.Ct[kk]);
          if (s.x0) t.x[k][q] = sqrt(D[k][q]) * s.x0[kk];
        }
      }
    __syncthreads();
    red[3] = res_delta0<double, KR>(t, R);
    ++c.tag;
    if (!(ok = res_allreduce<4>(red, c))) break;
    double gamma = red[0], delta = red[3];
    rr = red[1];
    bnorm = sqrt(red[2]);
    double gamma_old = 1.0, e1 = 0.0, e2 = 0.0, e3 = 0.0, best = rr;
    int best_it = 0;
    bool stalled = false;
    it = 0;
    while (!res_converged(rr, bnorm, s.eps) && it < s.max_iter) {
      const double beta = it == 0 ? 0.0 : gamma / gamma_old;
      const double alpha = gamma / (delta + beta * (e1 + e2) + beta * beta * e3);
      ++it;
      ++c.tag;
      res_sweep<double, KR, true>(c, t, P, R, alpha, beta, it == 1, D, bx, by, ntx, nty, red);
      if (!(ok = res_allreduce<6>(red, c))) break;
      gamma_old = gamma;
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
    noconv = !stalled && !res_converged(rr, bnorm, s.eps);
    if (!stalled) break;
    fallback = 1;
  }
  if (ok) {
#pragma unroll
    for (int k = 0; k < KR; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
        if (res_in(s, i, j)) s.x[s.off + (long)j * s.pitch + i] = t.x[k][q] / sqrt(D[k][q]);
      }
    if (rank == 0 && threadIdx.x == 0) {
      s.sc->cg_iters = it_all;
      s.sc->cg_fallback = fallback;
      s.sc->cg_noconv = noconv;
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
// next residual reads its neighbours.  0 after an error, 1 when done, 2 when the
// refinement stalled and the FP64 solve must take over.
template <int KR>
__device__ __forceinline__ int res_mixed(const ResSys &s, double eps_inner, unsigned rank, unsigned nb, double *sm,
                                         ResShared *sh) {
  constexpr int TH = res_th(KR);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ntx = res_ntx(s.nx), nty = (s.ny + TH - 1) / TH;
  const int bx = (int)(rank % ntx), by = (int)(rank / ntx);
  const int i0 = bx * kResTW, j0 = by * TH;
  float *P = reinterpret_cast<float *>(sm), *R = P + (TH + 4) * kResPitch;
  ResCtx c;
  if (!res_enter(s, rank, nb, KR, sh, &c)) return 0;
  ResTile<float, KR> t;
  const double none[KR][2] = {};
  double xd[KR][2];
#pragma unroll
  for (int k = 0; k < KR; ++k)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + 2 * lane + q, j = j0 + wid * KR + k;
      xd[k][q] = s.x0 && res_in(s, i, j) ? s.x0[s.off + (long)j * s.pitch + i] : 0.0;
    }
  res_setup<float, KR>(s, c, i0, j0, s.eliminate, sm, t);
  double rr = 0.0, rr_prev = 0.0, bnorm = 0.0;
  int it_all = 0, ret = 2;
  for (int outer = 0; outer < kResMaxOuter; ++outer) {
    // r = b - A x in FP64, r~ = r/sqrt|Ct| in FP32
    double red[8] = {0, 0, 0, 0, 0, 0, 0, 0};
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
    __syncthreads();
    red[3] = res_delta0<float, KR>(t, R);
    ++c.tag;
    if (!res_allreduce<4>(red, c)) {
      ret = 0;
      break;
    }
    rr = red[1];
    if (outer == 0) bnorm = sqrt(red[2]);
    if (res_converged(rr, bnorm, s.eps)) {
      ret = 1;
      break;
    }
    if (outer > 0 && rr > 1e-2 * rr_prev) break;  // no tenfold gain: FP64 takes over
    rr_prev = rr;
    // A~ d~ = r~ until (r~, r~) fell by eps_inner^2
    double gamma = red[0], delta = red[3], gamma_old = 1.0, e1 = 0.0, e2 = 0.0, e3 = 0.0;
    const double stop = eps_inner * eps_inner * gamma;
#pragma unroll
    for (int k = 0; k < KR; ++k) t.x[k][0] = t.x[k][1] = 0.0f;
    int it = 0;
    bool ok = true;
    while (gamma > stop && it < s.max_iter) {
      const double beta = it == 0 ? 0.0 : gamma / gamma_old;
      const double alpha = gamma / (delta + beta * (e1 + e2) + beta * beta * e3);
      ++it;
      ++c.tag;
      res_sweep<float, KR, false>(c, t, P, R, (float)alpha, (float)beta, it == 1, none, bx, by, ntx, nty, red);
      if (!(ok = res_allreduce<5>(red, c))) break;
      gamma_old = gamma;
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
    __threadfence();
    ++c.tag;
    if (!res_allreduce<1>(red, c)) {
      ret = 0;
      break;
    }
    __threadfence();
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
  res_leave(s, c);
  return ret;
}

}  // namespace

}  // namespace frehd

#endif
