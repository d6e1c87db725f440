// Cluster multi-shift CG (sm_100a): a whole solve of a small graph in one launch, the gathered
// direction in shared memory.
//
// The R columns of a solve are independent recurrences, so they are cut into groups of CG
// columns and each group is solved by one thread-block cluster (or one CTA), from the
// right-hand side to the output, without waiting for any other.  What bounds an iteration of
// a small graph in the kernel-per-phase driver is not bytes but three dependent launches with
// a last-CTA reduction each and the latency of its gathers through L2 (40 us an iteration at
// n = 2,000, 58 us at n = 20,000, R = 16, FP64).  Here an iteration
// (realworld/polar_gpu.py:100-125) of the group's columns is
//   A  v = (M + tau_0 I) d on the CTA's rows, partial d.v       -> barrier 1, a = rr / d.v
//   B  r <- r - a v, history slot, partial r.r                  -> barrier 2, beta
//   C  d <- r + beta d, sent to the cluster's other CTAs        -> barrier 3
// with hardware cluster barriers, the per-CTA partial sums exchanged through distributed
// shared memory, and the composed deferred update of the pole iterates every kHist
// iterations.  Sums have a fixed order: results do not depend on scheduling.
//
// Why shared memory.  A random 8- or 16-byte gather costs an SM 1.7 clocks per lane through
// L2 (one tag look-up per row, whatever its width) and 0.13 from its own shared memory, so
// every CTA of a cluster holds the whole direction of its columns, n x CG values (up to 28,000
// rows in FP64 and 56,000 in FP32 at CG = 1), and computes its share of the rows.  With more
// than one CTA the new direction goes through global memory once per iteration (own part
// written, the others' read back, contiguous).
//
// Layout.  cl_order sorts the rows by degree, deals them round the cluster's CTAs and numbers
// every row by its place (CTA, slot).  A warp takes slices of 32 rows of up to kClLight
// neighbours (a lane each), 4 rows of up to kClMid (8 lanes each) or one wider row, which bounds
// its chain of gathers; a few very wide rows take the whole CTA (cl_order).  cl_fill writes the
// neighbour lists in places, 16 bits each, as one stream of chunks per warp: a chunk is four
// neighbours per lane (one 8-byte load), so that the next chunks are read ahead without
// looking at the slices.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "graph_ops.cuh"
#include "host_util.h"
#include "msolve_cl.h"
#include "solver_core.cuh"

namespace polar {

namespace {

constexpr int kClMaxCta = 16;    // CTAs per cluster at most (non-portable size)
constexpr int kClPoles = 16;     // poles per pass of the deferred update
constexpr int kClLight = 16;     // neighbours up to which a row takes a lane,
constexpr int kClMid = 256;      // 8 lanes; beyond, a warp
constexpr int kClWide = 2048;    // neighbours above which a row may take the whole CTA
constexpr int kClMidRows = 4;    // rows of a warp at 8 lanes each
constexpr int kClAhead = 3;      // chunks past the end of a warp's neighbour stream that it may read
constexpr int kItemD = 5 + kNC;  // doubles per (pole, column): z, zp, h, ip, pn, composed row
constexpr int kPoleWarp = 14;    // warps 14 and 15 advance the poles before they join the rows
constexpr int kOrderThreads = 1024;
constexpr int kClHead = 8;       // words per CTA of ClGraph::head

POLAR_D unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Barrier of the cluster's threads.  The aligned forms need every lane of a warp at the same
// instruction, so the warp joins up here: callers arrive from one-lane branches.
POLAR_D void cl_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Store to the same shared-memory variable of CTA `rank` of the cluster.
POLAR_D void cl_store(double* local, unsigned rank, double v) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(local);
  unsigned ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}

// Fixed part of the dynamic shared memory, for CG columns.
template <typename T, int CG>
struct ClShared {
  double xbuf[2][kClMaxCta][CG];  // partial sums of every CTA of the cluster: d.v, r.r
  double red[kWarps][CG];
  double mred[kWarps][CG];
  double rr[2][CG], stop[CG], ap[CG], bp[CG], ag[CG], be[CG], chi[CG];
  int act[2][CG], iters[CG], bad[CG];
  int pf[kClPoles * CG];
  alignas(16) double coef[kClPoles * CG * composed_row<double>()];
};

// Sum of the warps' partials `red` of this CTA to every CTA's xbuf[which], and the barrier.
template <typename T, int CG>
POLAR_D void cl_exchange(ClShared<T, CG>& S, int which, int cs, int rank) {
  __syncthreads();
  if ((int)threadIdx.x < CG * cs) {
    const int c = threadIdx.x % CG, dst = threadIdx.x / CG;
    double v[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v[w] = S.red[w][c];
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1)
#pragma unroll
      for (int w = 0; w < o; ++w) v[w] += v[w + o];
    if (cs == 1) S.xbuf[which][0][c] = v[0];
    else cl_store(&S.xbuf[which][rank][c], dst, v[0]);
  }
  if (cs == 1) __syncthreads();
  else cl_sync();
}

template <typename T, int CG>
POLAR_D double cl_sum(const ClShared<T, CG>& S, int which, int cs, int c) {
  if (cs == 1) return S.xbuf[which][0][c];
  double v[kClMaxCta];
#pragma unroll
  for (int k = 0; k < kClMaxCta; ++k) v[k] = k < cs ? S.xbuf[which][k][c] : 0.0;
#pragma unroll
  for (int o = kClMaxCta / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < o; ++k) v[k] += v[k + o];
  return v[0];
}

// Warp partials of the lanes' column sums -> S.red.
template <typename T, int CG>
POLAR_D void cl_red(ClShared<T, CG>& S, double (&acc)[CG]) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (int v = 0; v < CG; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int v = 0; v < CG; ++v) S.red[threadIdx.x >> 5][v] = acc[v];
}

// The composed deferred update (shifted_update_composed) of the CTA's active rows: thread item
// = (pole subset, row, column).  When the rows are few the poles are spread over the threads.
// Arithmetic, coefficients and X are FP64 in both precisions (mixed: P and the history are
// FP32): an FP32 X would be rounded 17 times per block at its full size, which is most of the
// iterates' error (2.8e-7 of X over 170 iterations; 0.9e-7 to 1.4e-7 this way).
template <typename T, int CG>
POLAR_D void cl_flush(const SolvePrm<T>& P, ClShared<T, CG>& S, int grp, int a0, int na, int nsteps, bool first,
                      bool final_pass) {
  constexpr int NR = composed_row<double>();
  const int p = P.p, nA = P.nA;
  int ps = 1;
  while (ps < kClPoles && na * CG * ps * 2 <= kBlock) ps *= 2;
  const int c = threadIdx.x % CG;
  const int sub = (threadIdx.x / CG) % ps;
  const int rthr = threadIdx.x / (CG * ps);
  const int rpp = kBlock / (CG * ps);
  const int colg = grp * CG + c;
  const double* cmp = P.cmp + (size_t)grp * p * CG * kNC;
  const int* pfl = P.pflag + (size_t)grp * p * CG;
  double* Xb = P.cl.X + (size_t)grp * p * nA * CG;
  T* Pb = P.Pb + (size_t)grp * p * nA * CG;
  const T* hist = P.hist + (size_t)grp * kHist * nA * CG;
  for (int j0 = 0; j0 < p; j0 += kClPoles) {
    const int pc = min(kClPoles, p - j0);
    __syncthreads();
    for (int i = threadIdx.x; i < pc * CG * kNC; i += kBlock) {
      const int t = i % kNC, jl = i / kNC;
      const int dst = t == 0 ? 2 * kHist : t == 1 ? 2 * kHist + 1
                    : t < 2 + kHist ? 2 * (t - 2) : 2 * (t - 2 - kHist) + 1;
      S.coef[jl * NR + dst] = nsteps > 0 ? __ldcg(cmp + ((size_t)j0 * CG + jl) * kNC + t) : 0.0;
    }
    for (int i = threadIdx.x; i < pc * CG; i += kBlock) S.pf[i] = nsteps > 0 ? __ldcg(pfl + j0 * CG + i) : 0;
    __syncthreads();
    for (int e = rthr; e < na; e += rpp) {
      const int a = a0 + e;
      double hv[kHist];
#pragma unroll
      for (int k = 0; k < kHist; ++k) hv[k] = k < nsteps ? (double)hist[((size_t)k * nA + a) * CG + c] : 0.0;
      const int ao = __ldg(P.cl.aorig + a);
      const double w0 = (first && colg < P.R) ? __ldg(P.W + (size_t)__ldg(P.active + ao) * P.ldw + colg) : 0.0;
      auto load = [&](int jl, double& x, double& pv, bool& on) {
        on = S.pf[jl * CG + c] != 0;
        const size_t o = ((size_t)(j0 + jl) * nA + a) * CG + c;
        x = first ? 0.0 : ((on || final_pass) ? Xb[o] : 0.0);
        pv = first ? w0 : (on ? (double)Pb[o] : 0.0);
      };
      auto apply = [&](int jl, double x, double pv, bool on) {
        if (!first && !final_pass && !on) return;
        const size_t o = ((size_t)(j0 + jl) * nA + a) * CG + c;
        if (on) {
          const double* cf = S.coef + (jl * CG + c) * NR;
          const double p0 = pv;
          x = fma(cf[2 * kHist], p0, x);
          pv = cf[2 * kHist + 1] * p0;
#pragma unroll
          for (int k = 0; k < kHist; ++k) {
            const double2 q = *reinterpret_cast<const double2*>(cf + 2 * k);
            x = fma(q.x, hv[k], x);
            pv = fma(q.y, hv[k], pv);
          }
        }
        if (final_pass) {
          if (colg < P.R) {
            const size_t oo = ((size_t)(j0 + jl) * nA + ao) * P.ldx + colg;
            if (P.x_f32) reinterpret_cast<float*>(P.Xout)[oo] = (float)x;
            else reinterpret_cast<double*>(P.Xout)[oo] = x;
          }
        } else {
          Xb[o] = x;
          Pb[o] = (T)pv;
        }
      };
      // two poles in flight ahead of the arithmetic
      double x0 = 0.0, p0 = 0.0, x1 = 0.0, p1 = 0.0;
      bool on0 = false, on1 = false;
      if (sub < pc) load(sub, x0, p0, on0);
      if (sub + ps < pc) load(sub + ps, x1, p1, on1);
      for (int jl = sub; jl < pc; jl += 2 * ps) {
        const double xa = x0, pa = p0, xb = x1, pb = p1;
        const bool oa = on0, ob = on1;
        if (jl + 2 * ps < pc) load(jl + 2 * ps, x0, p0, on0);
        if (jl + 3 * ps < pc) load(jl + 3 * ps, x1, p1, on1);
        apply(jl, xa, pa, oa);
        if (jl + ps < pc) apply(jl + ps, xb, pb, ob);
      }
    }
  }
}

// One iteration's pole recurrences of the CTA's items, one lane each (pole_step's arithmetic),
// after the column scalars: `cur` indexes the residual it led to, cur ^ 1 who took part.
template <typename T, int CG>
POLAR_D void cl_poles(const SolvePrm<T>& P, ClShared<T, CG>& S, double* item, int* live, int* pflag, int rank, int cs,
                      int slot, int cur, double shift, int lane0, int nlanes) {
  const int items = P.p * CG;
  for (int k = lane0; rank + k * cs < items; k += nlanes) {
    const int q = rank + k * cs;
    const int j = q / CG, c = q % CG;
    double* st = item + (size_t)k * kItemD;
    double* cq = st + 5;
    if (slot == 0) {
      cq[0] = 0.0;
      cq[1] = 1.0;
      for (int i = 0; i < 2 * kHist; ++i) cq[2 + i] = 0.0;
      pflag[k] = 0;
    }
    if (!live[k] || !S.act[cur ^ 1][c]) continue;
    const double theta = __ldg(P.tau + j) - shift;
    const double a = S.ag[c], be = S.be[c], chi = S.chi[c];
    const double z = st[0], zp = st[1];
    const double zn = z / (1.0 + a * theta + chi * (1.0 - z / zp));
    const double fac = zn / z;
    const double aj = a * fac;
    const double bj = be * fac * fac;
    for (int i = 0; i < slot; ++i) {
      const double di = cq[2 + kHist + i];
      cq[2 + i] += aj * di;
      cq[2 + kHist + i] = bj * di;
    }
    const double beta = cq[1];
    cq[0] += aj * beta;
    cq[1] = bj * beta;
    cq[2 + kHist + slot] = zn;
    const double rrn = S.rr[cur][c];
    if (P.track) {
      const double ipv = st[3], pnv = st[4];
      st[2] += 2.0 * aj * ipv + aj * aj * pnv;
      st[3] = bj * (ipv + aj * pnv);
      st[4] = zn * zn * rrn + bj * bj * pnv;
    }
    st[1] = z;
    st[0] = zn;
    if (fabs(zn) * sqrt(rrn) <= S.stop[c]) live[k] = 0;
    pflag[k] = 1;
  }
}

// acc += sum of w X over a wide row's list positions t0, t0 + step, ... (places in `ix`).
template <typename T, int CG, bool W>
POLAR_D void cl_wide(const T* D, const unsigned short* ix, const double* wt, int deg, int t0, int step,
                     double (&acc)[CG]) {
  constexpr int U = 4;
  for (int t = t0; t < deg; t += U * step) {
    int jj[U];
    double wv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      jj[u] = t + u * step < deg ? (int)__ldg(ix + t + u * step) : -1;
      wv[u] = W && jj[u] >= 0 ? __ldg(wt + t + u * step) : 1.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (jj[u] >= 0) {
        T xv[CG];
        vload<T, CG>(xv, D + jj[u] * CG);
#pragma unroll
        for (int v = 0; v < CG; ++v) acc[v] = W ? fma(wv[u], (double)xv[v], acc[v]) : acc[v] + (double)xv[v];
      }
  }
}

POLAR_HD size_t cl_al16(size_t x) { return (x + 15) & ~size_t(15); }

// Shared memory of one CTA: the fixed part, pole items, the direction (one zero row at its
// end) and, with OWN, the own-row vectors r, v and, in mixed precision, the direction's
// remainder; without OWN these live in the workspace.
template <typename T, int CG>
POLAR_HD size_t cl_off_item() { return cl_al16(sizeof(ClShared<T, CG>)); }
template <typename T, int CG>
POLAR_HD size_t cl_off_d(int cs, int p) {
  return cl_off_item<T, CG>() + cl_al16((size_t)((p * CG + cs - 1) / cs) * (kItemD * 8 + 8));
}
template <typename T, int CG>
POLAR_HD size_t cl_off_own(int cs, int LS, int p) {
  return cl_off_d<T, CG>(cs, p) + cl_al16(((size_t)cs * LS + 1) * CG * sizeof(T));
}
template <typename T, int CG>
POLAR_HD size_t cl_smem(int cs, int LS, int p, bool own) {
  return cl_off_own<T, CG>(cs, LS, p) + (own ? (size_t)LS * CG * (8 + sizeof(T) + (sizeof(T) == 4 ? 4 : 0)) : 0);
}

// One cluster's whole solve: column group `grp` of problem P.  Every shared array is taken
// from the dynamic shared memory here, so that its accesses stay in the shared address space.
template <typename T, int CG, bool W, bool OWN>
POLAR_D void cl_run(const SolvePrm<T>& P, const int grp) {
  extern __shared__ __align__(16) unsigned char cl_sm[];
  const ClGraph& C = P.cl;
  const polar_graph& g = P.g;
  const int nA = P.nA, cs = C.cs, LS = C.LS, rank = cs > 1 ? (int)cl_rank() : 0;
  const int items = P.p * CG;  // (pole, column) items of the cluster
  ClShared<T, CG>& S = *reinterpret_cast<ClShared<T, CG>*>(cl_sm);
  double* const item = reinterpret_cast<double*>(cl_sm + cl_off_item<T, CG>());  // kItemD doubles each, and flags
  int* const live = reinterpret_cast<int*>(item + (size_t)((items + cs - 1) / cs) * kItemD);
  int* const pflag = live + (items + cs - 1) / cs;
  T* const D = reinterpret_cast<T*>(cl_sm + cl_off_d<T, CG>(cs, P.p));
  unsigned char* const own = cl_sm + cl_off_own<T, CG>(cs, LS, P.p);
  const size_t wsp = ((size_t)grp * cs + rank) * LS * CG;  // workspace vectors: [group][place][CG]
  double* const Vr = OWN ? reinterpret_cast<double*>(own) : P.r + wsp;
  T* const Vv = OWN ? reinterpret_cast<T*>(own + (size_t)LS * CG * 8) : P.v + wsp;
  float* const Vlo = OWN ? reinterpret_cast<float*>(own + (size_t)LS * CG * (8 + sizeof(T))) : P.dlo + wsp;
  T* const DX = P.d + (size_t)grp * cs * LS * CG;  // exchange of the direction between CTAs
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int base = rank * LS;                   // places of this CTA's slots
  const int places = cs * LS;
  T* const Down = D + (size_t)base * CG;        // own rows
  T* const hist = P.hist + (size_t)grp * kHist * nA * CG;
  const double shift = __ldg(P.tau);
  // own rows by slot, degree descending: nw of the whole CTA, n32 of a warp, n8 of 8 lanes and
  // the light ones; slices of a warp each
  const int* const head = C.head + kClHead * rank;
  const int nw = __ldg(head), n32 = __ldg(head + 1), n8 = __ldg(head + 2);
  const int a0 = __ldg(head + 3), na = __ldg(head + 4);
  const int q8 = n32 + (n8 + kClMidRows - 1) / kClMidRows;  // slices before the light ones
  const int nit = q8 + (LS - nw - n32 - n8 + 31) / 32;
  const int2* const slices = C.slice + (size_t)rank * C.SL;

  auto load_d = [&](int s, double (&x)[CG]) {
    T hi[CG];
    vload<T, CG>(hi, Down + (size_t)s * CG);
#pragma unroll
    for (int v = 0; v < CG; ++v) x[v] = (double)hi[v];
    if (sizeof(T) == 4) {
      float lo[CG];
      vload<float, CG>(lo, Vlo + (size_t)s * CG);
#pragma unroll
      for (int v = 0; v < CG; ++v) x[v] += (double)lo[v];
    }
  };
  auto store_d = [&](int s, const double (&x)[CG]) {
    T hi[CG];
#pragma unroll
    for (int v = 0; v < CG; ++v) hi[v] = (T)x[v];
    vstore<T, CG>(Down + (size_t)s * CG, hi);
    if (cs > 1) vstore<T, CG>(DX + (size_t)(base + s) * CG, hi);
    if (sizeof(T) == 4) {
      float lo[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) lo[v] = (float)(x[v] - (double)hi[v]);
      vstore<float, CG>(Vlo + (size_t)s * CG, lo);
    }
  };
  // the other CTAs' parts of the direction, after the barrier that follows store_d
  auto collect = [&]() {
    constexpr int V = 16 / (int)sizeof(T);
    constexpr int U = 8;
    const int part = LS * CG / V;  // 16-byte pieces per CTA (LS is a multiple of 32)
    const int total = (cs - 1) * part;
    const int own = rank * part;
    using Vec = typename VecType<T, V>::type;
    const Vec* src = reinterpret_cast<const Vec*>(DX);
    Vec* dst = reinterpret_cast<Vec*>(D);
    for (int i0 = threadIdx.x; i0 < total; i0 += U * kBlock) {
      Vec t[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kBlock;
        if (i < total) t[u] = __ldcg(src + (i < own ? i : i + part));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kBlock;
        if (i < total) dst[i < own ? i : i + part] = t[u];
      }
    }
    __syncthreads();
  };

  // ---- start: r = d = W, r.r, column and pole state ----
  if ((int)threadIdx.x < CG) D[(size_t)places * CG + threadIdx.x] = T(0);
  {
    double acc[CG];
#pragma unroll
    for (int v = 0; v < CG; ++v) acc[v] = 0.0;
    for (int s = threadIdx.x; s < LS; s += kBlock) {
      const int row = __ldg(C.srow + base + s);
      double w[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) {
        const int cc = grp * CG + v;
        w[v] = row >= 0 && cc < P.R ? __ldg(P.W + (size_t)row * P.ldw + cc) : 0.0;
        acc[v] += w[v] * w[v];
      }
      T zero[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) zero[v] = T(0);
      vstore<double, CG>(Vr + (size_t)s * CG, w);
      vstore<T, CG>(Vv + (size_t)s * CG, zero);
      store_d(s, w);
    }
    cl_red(S, acc);
  }
  if (cs > 1) cl_sync();  // every CTA of the cluster runs before its shared memory is written
  cl_exchange(S, 1, cs, rank);
  if (cs > 1) collect();
  bool any;
  int bad = 0;
  {
    int on = 0;
    if ((int)threadIdx.x < CG) {
      const int c = threadIdx.x;
      const double rr = cl_sum(S, 1, cs, c);
      if (!isfinite(rr)) {
        atomicCAS(P.ctl + 1, 0, (int)POLAR_ERR_NONFINITE);
        on = 2;
      }
      on |= rr > 0.0 ? 1 : 0;
      S.rr[0][c] = rr;
      S.stop[c] = P.tol * sqrt(rr);
      S.ap[c] = 1.0;
      S.bp[c] = 0.0;
      S.act[0][c] = on & 1;
      S.bad[c] = 0;
      S.iters[c] = 0;
    }
    bad = __syncthreads_or(on & 2);
    any = __syncthreads_or(on & 1) != 0;
    for (int k = threadIdx.x; rank + k * cs < items; k += kBlock) {
      const int c = (rank + k * cs) % CG;
      double* st = item + (size_t)k * kItemD;
      st[0] = 1.0;
      st[1] = 1.0;
      st[2] = 0.0;
      st[3] = 0.0;
      st[4] = S.rr[0][c];
      live[k] = S.rr[0][c] > 0.0 ? 1 : 0;
      pflag[k] = 0;
    }
    __syncthreads();
  }

  long long it = 0;
  int flushes = 0, slot = 0, cur = 0;
  bool first = true;
  bool late = false;  // the previous iteration's poles are still to be advanced
  bool more = any && !bad && P.maxit > 0;
  while (more) {
    // ---- the previous iteration's poles (their scalars stand until barrier 1) ----
    if (late && warp >= kPoleWarp)
      cl_poles<T, CG>(P, S, item, live, pflag, rank, cs, slot - 1, cur, shift, threadIdx.x - 32 * kPoleWarp, kBlock - 32 * kPoleWarp);
    __syncwarp();
    // ---- A: v = (M + tau_0 I) d, d.v ----
    double dacc[CG];
#pragma unroll
    for (int v = 0; v < CG; ++v) dacc[v] = 0.0;
    // a row from its neighbour sum: added edges, diagonal, v and d.v
    auto finish = [&](int s, double dg, double (&acc)[CG]) {
      dg += shift;
      T xi[CG], y[CG];
      vload<T, CG>(xi, Down + (size_t)s * CG);
      if (g.nx > 0) {
        const int ix = __ldg(C.sx + base + s);
        if (ix >= 0) {
          const int b = __ldg(g.d_xoff + ix), e = __ldg(g.d_xoff + ix + 1);
          for (int k = b; k < e; ++k) {
            const double w = g.d_xwt ? __ldg(g.d_xwt + k) : 1.0;
            T xv[CG];
            vload<T, CG>(xv, D + (size_t)__ldg(C.place + __ldg(g.d_xnbr + k)) * CG);
#pragma unroll
            for (int v = 0; v < CG; ++v) acc[v] = fma(w, (double)xv[v], acc[v]);
            dg += w;
          }
        }
      }
#pragma unroll
      for (int v = 0; v < CG; ++v) {
        y[v] = (T)fma(dg, (double)xi[v], -acc[v]);
        dacc[v] += (double)xi[v] * (double)y[v];
      }
      vstore<T, CG>(Vv + (size_t)s * CG, y);
    };
    // rows of the whole CTA: position t of the list goes to thread t mod kBlock
    for (int k = 0; k < nw; ++k) {
      const int2 sl = __ldg(slices + k);
      double acc[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) acc[v] = 0.0;
      cl_wide<T, CG, W>(D, C.ell + sl.x, C.ellw + sl.x, sl.y, threadIdx.x, kBlock, acc);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int v = 0; v < CG; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
      if (lane == 0)
#pragma unroll
        for (int v = 0; v < CG; ++v) S.mred[warp][v] = acc[v];
      __syncthreads();
      if ((int)threadIdx.x == 0) {
#pragma unroll
        for (int v = 0; v < CG; ++v) {
          acc[v] = 0.0;
          for (int w = 0; w < kWarps; ++w) acc[v] += S.mred[w][v];
        }
        finish(k, __ldg(C.sdiag + base + k), acc);
      }
      __syncthreads();
    }
    // slices: the warp's stream of chunks, two read ahead; one loop per kind of slice, in which
    // a lane's row advances by a constant stride
    if (warp < nit) {
      int q = warp, lens = 0;
      const uint2* cp = reinterpret_cast<const uint2*>(C.ell) + (size_t)__ldg(&slices[nw + warp].x) * 32 + lane;
      const double2* wp = reinterpret_cast<const double2*>(C.ellw + (cp - reinterpret_cast<const uint2*>(C.ell)) * 4);
      uint2 x0 = __ldg(cp), x1 = __ldg(cp + 32);
      cp += 64;
      double acc[CG], odd[CG];
      // sum of slice q's neighbours in acc, its chunk count from the warp's list (32 at a time)
      auto sum_slice = [&]() {
        const int i = q / kWarps;
        if ((i & 31) == 0) lens = q + kWarps * lane < nit ? __ldg(&slices[nw + q + kWarps * lane].y) : 1;
        int rem = __shfl_sync(0xffffffffu, lens, i & 31);
#pragma unroll
        for (int v = 0; v < CG; ++v) acc[v] = odd[v] = 0.0;
        do {
          T xv[4][CG];
          vload<T, CG>(xv[0], D + (x0.x & 0xffffu) * CG);
          vload<T, CG>(xv[1], D + (x0.x >> 16) * CG);
          vload<T, CG>(xv[2], D + (x0.y & 0xffffu) * CG);
          vload<T, CG>(xv[3], D + (x0.y >> 16) * CG);
          x0 = x1;
          x1 = __ldg(cp);
          cp += 32;
          if (W) {
            const double2 w0 = __ldg(wp), w1 = __ldg(wp + 1);
            wp += 64;
#pragma unroll
            for (int v = 0; v < CG; ++v) {
              acc[v] = fma(w0.x, (double)xv[0][v], acc[v]);
              odd[v] = fma(w0.y, (double)xv[1][v], odd[v]);
              acc[v] = fma(w1.x, (double)xv[2][v], acc[v]);
              odd[v] = fma(w1.y, (double)xv[3][v], odd[v]);
            }
          } else {
#pragma unroll
            for (int v = 0; v < CG; ++v) {
              acc[v] += (double)xv[0][v];
              odd[v] += (double)xv[1][v];
              acc[v] += (double)xv[2][v];
              odd[v] += (double)xv[3][v];
            }
          }
        } while (--rem > 0);
#pragma unroll
        for (int v = 0; v < CG; ++v) acc[v] += odd[v];
      };
      auto fold = [&](int per) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
          if (o < per)
#pragma unroll
            for (int v = 0; v < CG; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
      };
      for (; q < n32; q += kWarps) {
        const double dg = __ldg(C.sdiag + base + nw + q);
        sum_slice();
        fold(32);
        if (lane == 0) finish(nw + q, dg, acc);
      }
      for (; q < q8; q += kWarps) {
        const int s = nw + n32 + kClMidRows * (q - n32) + (lane >> 3);
        const bool ok = (lane & 7) == 0 && s < nw + n32 + n8;
        const double dg = ok ? __ldg(C.sdiag + base + s) : 0.0;
        sum_slice();
        fold(8);
        if (ok) finish(s, dg, acc);
      }
      int s = nw + n32 + n8 + 32 * (q - q8) + lane;
      const double* dp = C.sdiag + base + s;
      double dg = q < nit && s < LS ? __ldg(dp) : 0.0;
      for (; q < nit; q += kWarps, s += 32 * kWarps) {
        dp += 32 * kWarps;
        const double dn = s + 32 * kWarps < LS ? __ldg(dp) : 0.0;
        sum_slice();
        if (s < LS) finish(s, dg, acc);
        dg = dn;
      }
    }
    __syncwarp();
    cl_red(S, dacc);
    cl_exchange(S, 0, cs, rank);  // barrier 1
    int nf = 0;
    if ((int)threadIdx.x < CG) {
      const int c = threadIdx.x;
      const double a = S.act[cur][c] ? S.rr[cur][c] / cl_sum(S, 0, cs, c) : 0.0;
      if (!isfinite(a)) {
        atomicCAS(P.ctl + 1, 0, (int)POLAR_ERR_NONFINITE);
        nf = 1;
      }
      S.ag[c] = a;
    }
    bad |= __syncthreads_or(nf);
    // ---- B: r <- r - a v, history, r.r ----
    {
      double a_c[CG], racc[CG];
      bool on[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) {
        a_c[v] = S.ag[v];
        on[v] = S.act[cur][v] != 0;
        racc[v] = 0.0;
      }
      constexpr int U = CG == 1 ? 4 : 2;  // rows in flight per thread
      for (int s0 = threadIdx.x; s0 < LS; s0 += U * kBlock) {
        double rv[U][CG];
        T vv[U][CG];
        int ai[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int s = s0 + u * kBlock;
          if (s < LS) {
            ai[u] = __ldg(C.sact + base + s);
            vload<double, CG>(rv[u], Vr + (size_t)s * CG);
            vload<T, CG>(vv[u], Vv + (size_t)s * CG);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int s = s0 + u * kBlock;
          if (s >= LS) continue;
          T rt[CG];
#pragma unroll
          for (int v = 0; v < CG; ++v) {
            if (on[v]) rv[u][v] = rv[u][v] - a_c[v] * (double)vv[u][v];
            racc[v] += rv[u][v] * rv[u][v];
            rt[v] = (T)rv[u][v];
          }
          vstore<double, CG>(Vr + (size_t)s * CG, rv[u]);
          if (ai[u] >= 0) vstore<T, CG>(hist + ((size_t)slot * nA + ai[u]) * CG, rt);
        }
      }
      __syncwarp();
      cl_red(S, racc);
    }
    cl_exchange(S, 1, cs, rank);  // barrier 2
    // ---- column scalars, alike in every CTA: beta, convergence and chi on different warps ----
    if ((int)threadIdx.x < 96 && lane < CG) {
      const int c = lane;
      const int a_on = S.act[cur][c];
      const double rrn = cl_sum(S, 1, cs, c);
      if (warp == 0) {
        S.be[c] = a_on ? rrn / S.rr[cur][c] : 0.0;
        S.rr[cur ^ 1][c] = a_on ? rrn : S.rr[cur][c];
      } else if (warp == 1) {
        S.act[cur ^ 1][c] = a_on && sqrt(rrn) > S.stop[c];
        if (a_on) {
          S.iters[c] += 1;
          if (!isfinite(rrn)) {
            atomicCAS(P.ctl + 1, 0, (int)POLAR_ERR_NONFINITE);
            S.bad[c] = 1;
          }
        }
      } else if (a_on) {
        const double a = S.ag[c];
        S.chi[c] = a * S.bp[c] / S.ap[c];
        S.ap[c] = a;
        S.bp[c] = rrn / S.rr[cur][c];
      }
    }
    __syncthreads();
    any = false;
#pragma unroll
    for (int v = 0; v < CG; ++v) {
      any |= S.act[cur ^ 1][v] != 0;
      bad |= S.bad[v];
    }
    cur ^= 1;
    ++it;
    more = any && !bad && it < P.maxit;
    late = more && slot + 1 < kHist;
    if (!late) {
      // end of a block: the poles now, and their composed rows for the flush
      cl_poles<T, CG>(P, S, item, live, pflag, rank, cs, slot, cur, shift, threadIdx.x, kBlock);
      __syncthreads();
      for (int i = threadIdx.x; i < items * kNC; i += kBlock) {
        const int k = i / kNC, t = i % kNC;
        const int q = rank + k * cs;
        if (q >= items) break;
        P.cmp[((size_t)grp * items + q) * kNC + t] = item[(size_t)k * kItemD + 5 + t];
        if (t == 0) P.pflag[(size_t)grp * items + q] = pflag[k];
      }
    }
    // ---- C: d <- r + beta d ----
    if (more) {
      double be_c[CG];
      bool on[CG];
#pragma unroll
      for (int v = 0; v < CG; ++v) {
        be_c[v] = S.be[v];
        on[v] = S.act[cur ^ 1][v] != 0;
      }
      constexpr int U = CG == 1 ? 4 : 2;
      for (int s0 = threadIdx.x; s0 < LS; s0 += U * kBlock) {
        double rv[U][CG], dv[U][CG];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int s = s0 + u * kBlock;
          if (s < LS) {
            vload<double, CG>(rv[u], Vr + (size_t)s * CG);
            load_d(s, dv[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int s = s0 + u * kBlock;
          if (s >= LS) continue;
#pragma unroll
          for (int v = 0; v < CG; ++v)
            if (on[v]) dv[u][v] = rv[u][v] + be_c[v] * dv[u][v];
          store_d(s, dv[u]);
        }
      }
    }
    if (cs > 1) {  // barrier 3
      cl_sync();
      if (more) collect();
    } else {
      __syncthreads();
    }
    ++slot;
    if (more && slot == kHist) {
      cl_flush<T, CG>(P, S, grp, a0, na, slot, first, false);
      first = false;
      slot = 0;
      ++flushes;
    }
  }
  // ---- remaining steps, X -> output ----
  cl_flush<T, CG>(P, S, grp, a0, na, slot, first, true);
  if (P.track && P.h_out)
    for (int k = threadIdx.x; rank + k * cs < items; k += kBlock) {
      const int q = rank + k * cs, j = q / CG, cc = grp * CG + q % CG;
      if (cc < P.R) P.h_out[(size_t)j * P.R + cc] = item[(size_t)k * kItemD + 2];
    }
  if (rank == 0 && (int)threadIdx.x < CG && grp * CG + (int)threadIdx.x < P.R)
    P.iters_out[grp * CG + threadIdx.x] = S.iters[threadIdx.x];
  if (rank == 0 && threadIdx.x == 0) {
    atomicMax(P.stats, it);
    atomicMax(P.stats + 1, (long long)(flushes + 1));
    if (any && it >= P.maxit) atomicMax(P.ctl, (int)POLAR_ERR_ITER_CAP);
  }
}

template <typename T, int CG, bool W, bool OWN>
__global__ void __launch_bounds__(kBlock, 1) cl_solve(const __grid_constant__ SolvePrm<T> P) {
  cl_run<T, CG, W, OWN>(P, blockIdx.x / P.cl.cs);
}

// ---- row order, places and neighbour lists of one problem -----------------------------------
POLAR_D int cl_key(const polar_graph& g, int row) {
  const int deg = __ldg(g.d_indptr + row + 1) - __ldg(g.d_indptr + row);
  // degree descending in classes that part kClLight, kClMid and the powers of two from 1,024: one
  // per degree up to 64, then by 8 up to 512, by 32 up to 1,024 and by doubling
  const int c = deg <= 64     ? deg
                : deg <= 512  ? 64 + (deg - 57) / 8
                : deg <= 1024 ? 121 + (deg - 481) / 32
                              : 128 + (31 - __clz(deg - 1));
  return 255 - c;
}

// Exclusive scan of one int per thread over the block; returns the thread's prefix, total in *sum.
POLAR_D int block_scan(int x, int* tmp, int* sum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  __syncthreads();
  if (lane == 31) tmp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int w = tmp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    tmp[32 + lane] = w;
  }
  __syncthreads();
  *sum = tmp[63];
  return v - x + (warp ? tmp[31 + warp] : 0);
}

// One CTA: rows sorted by degree class (stable radix sort, two passes of four bits, each
// thread a contiguous piece), then slots, slices, hubs and the order of the active rows.
__global__ void __launch_bounds__(kOrderThreads) cl_order(polar_graph g, ClGraph C, const int* active_pos) {
  extern __shared__ int cnt[];  // 16 x kOrderThreads
  __shared__ int tmp[64];
  __shared__ int over[5];  // rows of more than kClWide << k neighbours
  const int n = g.n, t = threadIdx.x;
  const int per = (n + kOrderThreads - 1) / kOrderThreads;
  const int lo = min(n, t * per), hi = min(n, lo + per);
  for (int pass = 0; pass < 2; ++pass) {
    const int* src = pass == 0 ? nullptr : C.tmp0;
    int* dst = pass == 0 ? C.tmp0 : C.tmp1;
    for (int d = 0; d < 16; ++d) cnt[d * kOrderThreads + t] = 0;
    for (int i = lo; i < hi; ++i) {
      const int row = src ? src[i] : i;
      cnt[((cl_key(g, row) >> (4 * pass)) & 15) * kOrderThreads + t] += 1;
    }
    __syncthreads();
    // exclusive scan over (digit, thread): thread t scans 16 consecutive counters
    int s = 0, sum;
    for (int k = 0; k < 16; ++k) s += cnt[t * 16 + k];
    int p = block_scan(s, tmp, &sum);
    __syncthreads();
    for (int k = 0; k < 16; ++k) {
      const int c = cnt[t * 16 + k];
      cnt[t * 16 + k] = p;
      p += c;
    }
    __syncthreads();
    for (int i = lo; i < hi; ++i) {
      const int row = src ? src[i] : i;
      dst[cnt[((cl_key(g, row) >> (4 * pass)) & 15) * kOrderThreads + t]++] = row;
    }
    __syncthreads();
  }
  const int* order = C.tmp1;
  const int cs = C.cs, LS = C.LS, places = cs * LS;
  auto degree = [&](int row) { return g.d_indptr[row + 1] - g.d_indptr[row]; };
  for (int i = t; i < places; i += kOrderThreads) {
    C.srow[i] = -1;
    C.sx[i] = -1;
    C.sdiag[i] = 0.0;
  }
  // rows above the limits of 8 lanes and one lane
  if (t < 5) over[t] = 0;
  __syncthreads();
  int nh = 0, nm = 0;
  for (int i = lo; i < hi; ++i) {
    const int deg = degree(order[i]);
    nh += deg > kClMid;
    nm += deg > kClLight;
    for (int k = 0; k < 5 && deg > kClWide << k; ++k) atomicAdd(&over[k], 1);
  }
  __syncthreads();
  // Rows of the whole CTA.  One costs all its warps two barriers and a serial sum, 1,500 clocks, and
  // a clock per 14 neighbours; on a warp it is 0.7 clock per neighbour, the other warps having
  // rows of their own.  So rows of more than L neighbours are taken by the CTA when its w of them
  // are cheaper than one on a warp: from 4,096 when it has one, never from six on.  FP64 solves,
  // rows of more than 1,024 on the CTA -> this: 2,500 rows of 1,100 neighbours R = 1 2.19 -> 0.98 ms;
  // n = 20,000 with 50 rows of 5,000 R = 16 6.28 -> 5.14, with 300 of 1,200 7.51 -> 4.65.
  int nwide = 0;
  for (int k = 0; k < 5; ++k) {
    const int L = kClWide << k, w = (over[k] + cs - 1) / cs;
    if (w * (1500 + L / 14) < 0.7 * L) {
      nwide = over[k];
      break;
    }
  }
  int nhub, nmid;
  block_scan(nh, tmp, &nhub);
  block_scan(nm, tmp, &nmid);
  __syncthreads();
  for (int i = lo; i < hi; ++i) {  // row i of the order: slot i / cs of CTA i % cs
    const int row = order[i];
    const int place = (i % cs) * LS + i / cs;
    C.place[row] = place;
    C.srow[place] = row;
    C.sdiag[place] = g.d_diag ? g.d_diag[row] : (double)degree(row) + g.sigma;
    if (g.nx > 0 && (g.d_xbits[row >> 5] >> (row & 31)) & 1u) {
      int a = 0, b = g.nx - 1;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (g.d_xrow[mid] < row) a = mid + 1;
        else b = mid;
      }
      C.sx[place] = a;
    }
  }
  __syncthreads();
  // Chunks of every slice (from its longest row; at least one), then where each warp's stream
  // and each wide row's list starts.
  for (int r = 0; r < cs; ++r) {
    auto upto = [&](int m) { return m > r ? (m - r + cs - 1) / cs : 0; };  // rows of CTA r among the first m
    const int w = upto(nwide), h = upto(nhub), m = upto(nmid);
    const int q8 = h + (m - h + kClMidRows - 1) / kClMidRows;
    const int total = q8 + (LS - m + 31) / 32;
    for (int k = t; k < total; k += kOrderThreads) {
      const int s = k < h ? k : k < q8 ? h + kClMidRows * (k - h) : m + 32 * (k - q8);
      // light rows are in exact order, the others in classes
      int deg = 0;
      for (int e = 0; e < (k >= h && k < q8 ? kClMidRows : 1); ++e) {
        const int row = s + e < LS ? C.srow[r * LS + s + e] : -1;
        if (row >= 0) deg = max(deg, degree(row));
      }
      const int lanes = k < h ? 32 : k < q8 ? 8 : 1;
      C.slice[r * C.SL + k] = make_int2(0, k < w ? deg : max(1, (deg + 4 * lanes - 1) / (4 * lanes)));
    }
    if (t == 0) {
      C.head[kClHead * r] = w;
      C.head[kClHead * r + 1] = h - w;
      C.head[kClHead * r + 2] = m - h;
      C.head[kClHead * r + 5] = total;
    }
  }
  __syncthreads();
  int off;
  {
    const int r = t / kWarps, wp = t % kWarps;  // warp wp of CTA r
    const int w = r < cs ? C.head[kClHead * r] : 0, total = r < cs ? C.head[kClHead * r + 5] : 0;
    int2* const sl = C.slice + (size_t)r * C.SL;
    int len = 0;
    for (int k = w + wp; k < total; k += kWarps) len += sl[k].y;
    int o = block_scan(len, tmp, &off);
    for (int k = w + wp; k < total; k += kWarps) {
      sl[k].x = o;
      o += sl[k].y;
    }
  }
  off = (off + kClAhead) * 128;  // list entries, with the chunks that a stream's end reads ahead
  for (int i = t; i < nwide; i += kOrderThreads) {  // wide rows are few: each sums the ones before it
    int o = off;
    for (int k = 0; k < i; ++k) o += (degree(order[k]) + 7) & ~7;
    C.slice[(size_t)(i % cs) * C.SL + i / cs].x = o;
  }
  // active rows in the order of their places
  const int pp = (places + kOrderThreads - 1) / kOrderThreads;
  const int plo = min(places, t * pp), phi = min(places, plo + pp);
  __syncthreads();
  int na = 0, sum;
  for (int i = plo; i < phi; ++i) na += C.srow[i] >= 0 && active_pos[C.srow[i]] >= 0;
  int a = block_scan(na, tmp, &sum);
  for (int i = plo; i < phi; ++i) {
    if (i % LS == 0) C.head[kClHead * (i / LS) + 3] = a;
    const int row = C.srow[i];
    const int ap = row >= 0 ? active_pos[row] : -1;
    C.sact[i] = ap >= 0 ? a : -1;
    if (ap >= 0) C.aorig[a++] = ap;
  }
  __syncthreads();
  if (t < cs) C.head[kClHead * t + 4] = (t + 1 < cs ? C.head[kClHead * t + kClHead + 3] : sum) - C.head[kClHead * t + 3];
}

// Neighbour lists in places: one warp per hub or slice of a CTA's rows.
template <bool W>
__global__ void cl_fill(polar_graph g, ClGraph C) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const int LS = C.LS;
  const unsigned short pad = (unsigned short)(C.cs * LS);  // the zero row
  for (int r = 0; r < C.cs; ++r) {
    const int w = C.head[kClHead * r], h = w + C.head[kClHead * r + 1], m = h + C.head[kClHead * r + 2];
    const int q8 = h + (m - h + kClMidRows - 1) / kClMidRows;
    const int total = q8 + (LS - m + 31) / 32;
    for (int k = (wid + r * 7) % nw; k < total; k += nw) {
      const int2 sl = C.slice[r * C.SL + k];
      if (k < w) {
        const int lo = g.d_indptr[C.srow[r * LS + k]];
        for (int t = lane; t < sl.y; t += 32) {
          C.ell[sl.x + t] = (unsigned short)C.place[g.d_indices[lo + t]];
          if (W) C.ellw[sl.x + t] = g.d_wts[lo + t];
        }
        continue;
      }
      const int lanes = k < h ? 32 : k < q8 ? 8 : 1;
      const int s = k < h ? k : k < q8 ? h + kClMidRows * (k - h) + (lane >> 3) : m + 32 * (k - q8) + lane;
      const int row = s < (k < q8 ? m : LS) ? C.srow[r * LS + s] : -1;
      int lo = 0, deg = 0;
      if (row >= 0) {
        lo = g.d_indptr[row];
        deg = g.d_indptr[row + 1] - lo;
      }
      for (int t = 0; t < 4 * sl.y; ++t) {
        const size_t o = ((size_t)(sl.x + (t >> 2)) * 32 + lane) * 4 + (t & 3);
        const int e = (lane & (lanes - 1)) + lanes * t;
        C.ell[o] = e < deg ? (unsigned short)C.place[g.d_indices[lo + e]] : pad;
        if (W) C.ellw[o] = e < deg ? g.d_wts[lo + e] : 0.0;
      }
    }
  }
}

constexpr size_t kClSmemMax = 232448;  // 227 KB

// Launch shape of a solve: columns per cluster, CTAs per cluster and what its rows keep on chip.
struct ClPlan {
  int cg = 0, cs = 0, groups = 0, LS = 0;
  bool own = false;
  size_t smem = 0;
  double cost = 1e300;  // clocks per iteration
};

template <typename F>
cudaError_t cl_attributes(F* fn) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmemMax);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

// Clusters of cs CTAs, one CTA per SM, that the device holds at a time (0: none).
struct ClResident {
  int most[kClMaxCta + 1] = {0};
  ClResident() {
    if (cl_attributes(cl_solve<double, 1, false, false>) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    for (int cs = 1; cs <= kClMaxCta; ++cs) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(cs);
      cfg.blockDim = dim3(kBlock);
      cfg.dynamicSmemBytes = kClSmemMax;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = cs;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&most[cs], cl_solve<double, 1, false, false>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        most[cs] = 0;
      }
    }
  }
};

// Whether this thread's solves may take the cluster kernel.
thread_local bool g_cluster = true;

int cl_resident(int cs) {
  static const ClResident r;
  return r.most[cs];
}

// What the choice of a launch shape depends on.
struct ClShape {
  int n, nnz, nx;
  bool weighted;
  int R, ld, p, nA;
};

template <typename T, int CG>
void cl_try(const ClShape& S, int cs, ClPlan& best) {
  ClPlan s;
  s.cg = CG;
  s.cs = cs;
  s.groups = (S.R + CG - 1) / CG;
  s.LS = ((S.n + cs - 1) / cs + 31) / 32 * 32;
  const int most = cl_resident(cs);
  if (most < 1 || (long long)cs * s.LS + 1 > 65536 || (long long)cs * s.LS > S.n + kClPad) return;
  s.own = cl_smem<T, CG>(cs, s.LS, S.p, true) <= kClSmemMax;
  s.smem = cl_smem<T, CG>(cs, s.LS, S.p, s.own);
  if (s.smem > kClSmemMax) return;
  // Clocks per iteration, for the choice between launch shapes, fitted to solves of 2,000 to 57,000
  // rows with 4 to 18 neighbours: fixed reductions and scalars; gathers; the CTA's rows, dearer
  // when their vectors come from L2; the deferred update; with several CTAs their barriers and
  // the direction's exchange.
  const double rows = (double)S.n / cs;
  double c = 5000 + (0.25 + 0.02 * CG * sizeof(T) + (S.weighted ? 0.3 : 0.0)) * S.nnz / cs + rows * CG * (s.own ? 3.0 : 4.5) +
             0.015 * sizeof(T) * CG * (double)S.nA * S.p / cs;
  if (cs > 1) c += 4000 + (double)S.n * CG * sizeof(T) / 30.0;
  s.cost = c * std::max(1.0, std::ceil((double)s.groups / most));
  if (s.cost < best.cost) best = s;
}

template <typename T>
ClPlan cl_plan(const ClShape& S) {
  ClPlan best;
  for (int cs = 1; cs <= kClMaxCta; ++cs) {
    cl_try<T, 1>(S, cs, best);
    if (S.ld >= 2) cl_try<T, 2>(S, cs, best);
    if (sizeof(T) == 4 && S.ld >= 4) cl_try<T, 4>(S, cs, best);
  }
  return best;
}

template <typename T, int CG, bool W, bool OWN>
cudaError_t cl_launch(const SolvePrm<T>& P, const ClPlan& s, cudaStream_t st) {
  cudaError_t e = cl_attributes(cl_solve<T, CG, W, OWN>);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(s.groups * s.cs);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = s.cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, cl_solve<T, CG, W, OWN>, P);
}

template <typename T, int CG>
cudaError_t cl_launch(const SolvePrm<T>& P, const ClPlan& s, cudaStream_t st) {
  if (P.g.d_wts) return s.own ? cl_launch<T, CG, true, true>(P, s, st) : cl_launch<T, CG, true, false>(P, s, st);
  return s.own ? cl_launch<T, CG, false, true>(P, s, st) : cl_launch<T, CG, false, false>(P, s, st);
}

template <typename T>
cudaError_t cl_launch(const SolvePrm<T>& P, const ClPlan& s, cudaStream_t st) {
  if constexpr (sizeof(T) == 4)
    if (s.cg == 4) return cl_launch<T, 4>(P, s, st);
  return s.cg == 2 ? cl_launch<T, 2>(P, s, st) : cl_launch<T, 1>(P, s, st);
}

}  // namespace

size_t cl_graph_bytes(const polar_graph* g, int nA) {
  ClGraph C;
  return cl_graph_layout(g, nA, nullptr, &C);
}

size_t cl_graph_layout(const polar_graph* g, int nA, char* base, ClGraph* C) {
  size_t o = 0;
  auto take = [&](size_t bytes) {
    char* p = base + o;
    o += (bytes + 255) & ~size_t(255);
    return p;
  };
  // List entries.  A slice of the longest row d takes 128 ceil(d / 4L) entries, L lanes per row:
  // at most 32 d + 96 for 32 light rows, 4 d + 124 for 4 rows of more than 16 neighbours and
  // d + 127 for a row of more than 256.  Along a CTA's slices d falls (by classes of at most an
  // eighth), so these sum to less than 3 nnz + 3 n and, per CTA, the first slice of each kind;
  // then the chunks read ahead at the end.
  const size_t n = g->n, places = n + kClPad;
  const size_t ell = 3 * (size_t)g->nnz + 4 * n + (size_t)kClMaxCta * 4096 + 4 * kClPad;
  C->tmp0 = (int*)take(n * 4);
  C->tmp1 = (int*)take(n * 4);
  C->place = (int*)take(n * 4);
  C->srow = (int*)take(places * 4);
  C->sact = (int*)take(places * 4);
  C->sx = (int*)take(places * 4);
  C->sdiag = (double*)take(places * 8);
  C->aorig = (int*)take((size_t)nA * 4);
  C->slice = (int2*)take((places + 2 * kClMaxCta) * 8);
  C->head = (int*)take(kClHead * kClMaxCta * 4);
  C->ell = (unsigned short*)take(ell * 2);
  C->ellw = (double*)take(g->d_wts ? ell * 8 : 0);
  return o;
}

// Which driver is the faster one, from clocks per iteration of either, fitted (least squares of the
// ratio) to 8,700 solves of 1,500 to 58,000 rows with 4 to 18 neighbours, 1 to 128 columns, 44 % of
// them with added edges.  Cluster: its fixed part (more with several CTAs), gathers, the CTA's
// rows (dearer when their vectors come from L2), the deferred update, the direction's exchange,
// added edges; as often as its clusters need turns.  Kernels per phase: launches, reductions and
// gather latency, their vectors, and mk_added's launch or the SpMM's tail.  Of the solves 98.4 %
// end up with the faster driver to 3 % (worst 1.27x); without terms for added edges 3 % of them
// took the cluster solver though it was slower, by up to 1.7x (n = 28,000 R = 64 FP64 with added
// edges in 3,900 rows: 113 us an iteration, 82 by phases).
template <typename T>
static bool cl_faster(const ClShape& S) {
  const ClPlan b = cl_plan<T>(S);
  if (b.groups == 0) return false;
  const double rows = (double)S.n / b.cs, es = sizeof(T), own = b.own ? 1.7 : es == 8 ? 2.1 : 2.8;
  double here = 6700 + (0.45 + (S.weighted ? 0.12 : 0.0)) * S.nnz / b.cs + rows * b.cg * own +
                0.02 * es * b.cg * (double)S.nA * S.p / b.cs;
  if (b.cs > 1) here += 6700 + 0.04 * es * b.cg * S.n;
  if (S.nx > 0) here += 3200 + 20.0 * S.nx / b.cs;
  here *= std::max(1.0, std::ceil((double)b.groups / cl_resident(b.cs)));
  double phases = 75000 + 63 * es * S.ld + 0.018 * S.nnz + 0.02 * (double)S.ld * S.n;
  if (S.weighted) phases += 11300 + 0.009 * S.nnz;
  if (S.nx > 0) phases += added_split(S.nx, S.ld) ? 13000 + 0.04 * (double)S.nx * S.ld : 3300;
  return here < phases;
}

bool cl_takes(const polar_graph* g, int precision, int R, int ld, int p, int nA) {
  if (!g_cluster || g->n > kClMaxRows) return false;
  const ClShape S{g->n, g->nnz, g->nx, g->d_wts != nullptr, R, ld, p, nA};
  return precision == POLAR_MIXED ? cl_faster<float>(S) : cl_faster<double>(S);
}

template <typename T>
int cl_solve_one(const SolvePrm<T>& P0, cudaStream_t st, MkResult* out) {
  SolvePrm<T> P = P0;
  const ClPlan s = cl_plan<T>(ClShape{P.g.n, P.g.nnz, P.g.nx, P.g.d_wts != nullptr, P.R, P.ld, P.p, P.nA});
  P.cl.cs = s.cs;
  P.cl.LS = s.LS;
  P.cl.SL = s.LS + 2;
  const bool w = P.g.d_wts != nullptr;
  const size_t osm = 16 * kOrderThreads * sizeof(int);
  cudaError_t e = cudaFuncSetAttribute(cl_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)osm);
  if (e != cudaSuccess) return set_cuda_error("cl_order", e);
  cl_order<<<1, kOrderThreads, osm, st>>>(P.g, P.cl, P.active_pos);
  const int fill = std::min(296, (P.g.n / 32 + 8) / 8 + 1);
  if (w) cl_fill<true><<<fill, 256, 0, st>>>(P.g, P.cl);
  else cl_fill<false><<<fill, 256, 0, st>>>(P.g, P.cl);
  e = cudaGetLastError();
  TimedLaunch t{KC_CLUSTER, 0.0, nullptr, nullptr};
  const bool timing = timing_on();
  if (timing) {
    t.a = timing_event();
    t.b = timing_event();
    cudaEventRecord(t.a, st);
  }
  if (e == cudaSuccess) e = cl_launch(P, s, st);
  count_launch(3);
  if (timing) {
    cudaEventRecord(t.b, st);
    timing_push(t);
  }
  if (e != cudaSuccess) return set_cuda_error("cl_solve", e);
  int ctl[2] = {0, 0};
  long long stats[2] = {0, 0};
  e = cudaMemcpyAsync(ctl, P.ctl, sizeof(ctl), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(stats, P.stats, sizeof(stats), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return set_cuda_error("cl_solve", e);
  if (timing) timing_collect();
  out->err = ctl[1];
  out->capped = ctl[1] == 0 && ctl[0] != 0;
  out->iterations = stats[0];
  out->flushes = stats[1];
  out->grid = s.groups * s.cs;
  return POLAR_OK;
}

template int cl_solve_one<float>(const SolvePrm<float>&, cudaStream_t, MkResult*);
template int cl_solve_one<double>(const SolvePrm<double>&, cudaStream_t, MkResult*);

}  // namespace polar

extern "C" int polar_set_cluster_solver(int on) {
  const int was = polar::g_cluster ? 1 : 0;
  polar::g_cluster = on != 0;
  return was;
}
