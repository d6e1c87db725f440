// Greedy-round kernels of POLAR (sm_100a): incidence right-hand sides, bank caches,
// proxy score + stable top-B, re-rank, Sherman–Morrison maintenance and the F update.
// All are HBM-bound gathers/streams; they keep every selection on the device, so a
// round needs one small device->host read (the winner) and nothing else.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "host_util.h"

namespace polar {

template <typename T>
POLAR_D double ldx(const void* p, size_t i) {
  return (double)reinterpret_cast<const T*>(p)[i];
}
POLAR_D double ldv(const void* p, int f32, size_t i) { return f32 ? ldx<float>(p, i) : ldx<double>(p, i); }

POLAR_HD size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// ---------------------------------------------------------------------------------------
// W[:, c] = e_a - e_b with (a, b) = cand[sel[c]]; ia/ib = endpoint active positions.
__global__ void fill_incidence_kernel(int R, const int64_t* cand, const int64_t* sel, const int32_t* es,
                                      double* W, int ldw, int32_t* ia, int32_t* ib) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= R) return;
  const int64_t e = sel[c];
  W[(size_t)cand[2 * e] * ldw + c] = 1.0;
  W[(size_t)cand[2 * e + 1] * ldw + c] = -1.0;
  if (ia) ia[c] = es[2 * e];
  if (ib) ib[c] = es[2 * e + 1];
}

// ---------------------------------------------------------------------------------------
// out[j][e] = sum_c (X[j][ea][col0+c] - X[j][eb][col0+c])^2 ; 16 lanes per (j, e).
template <typename T>
__global__ void pair_norms_kernel(const T* X, int p, int nA, int ldx, int col0, int q, const int32_t* ea,
                                  const int32_t* eb, int N, double* out) {
  const int lanes = 16;
  const long long gidx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / lanes;
  const int lg = threadIdx.x & (lanes - 1);
  const unsigned mask = 0xffffu << (threadIdx.x & 16);
  const long long total = (long long)p * N;
  if (gidx >= total) return;
  const int j = (int)(gidx / N), e = (int)(gidx % N);
  const T* xa = X + ((size_t)j * nA + ea[e]) * ldx + col0;
  const T* xb = X + ((size_t)j * nA + eb[e]) * ldx + col0;
  double s = 0.0;
  for (int c = lg; c < q; c += lanes) {
    const double dlt = (double)xa[c] - (double)xb[c];
    s += dlt * dlt;
  }
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
  if (lg == 0) out[(size_t)j * N + e] = s;
}

// ---------------------------------------------------------------------------------------
// Stable top-B: key order (score descending, index ascending).
POLAR_D bool better(double s1, long long i1, double s2, long long i2) {
  return s1 > s2 || (s1 == s2 && i1 < i2);
}

constexpr int kTopBlock = 256;  // candidates per CTA of the scoring pass
constexpr int kMergeBlock = 1024;
constexpr int kMaxB = 64;

struct Cand {
  double s;
  long long i;
};

POLAR_D Cand warp_best(Cand c) {
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_xor_sync(0xffffffffu, c.s, o);
    const long long i2 = __shfl_xor_sync(0xffffffffu, c.i, o);
    if (better(s2, i2, c.s, c.i)) {
      c.s = s2;
      c.i = i2;
    }
  }
  return c;
}

// Block-wide argmax by (score, index); all threads get the result.
POLAR_D Cand block_best(Cand c, Cand* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  c = warp_best(c);
  if (lane == 0) sh[warp] = c;
  __syncthreads();
  if (warp == 0) {
    Cand d = lane < (int)(blockDim.x >> 5) ? sh[lane] : Cand{-INFINITY, LLONG_MAX};
    d = warp_best(d);
    if (lane == 0) sh[32] = d;
  }
  __syncthreads();
  Cand r = sh[32];
  __syncthreads();
  return r;
}

// Scores of one candidate per thread, kept in `score`, and each CTA's best live one.  The pass
// is bound by its 16 p N bytes of caches: the poles are taken four at a time so that enough
// loads are in flight, and a CTA reduces once (not B times: the B best of a million candidates
// at p = 32, B = 16 took 199 us that way, 78 us being the caches' bytes; this pass and the
// merge take 91 and 28).
template <int OBJ>
__global__ void __launch_bounds__(kTopBlock, 4) score_kernel(const double* h, const double* t, const double* tau,
                                                          const double* om, double sigma, int p, int N,
                                                          const uint8_t* live, double* score, Cand* best) {
  __shared__ Cand sh[33];
  const long long e = (long long)blockIdx.x * kTopBlock + threadIdx.x;
  Cand mine{-INFINITY, LLONG_MAX};
  if (e < N) {
    double v;
    if (OBJ == 1) {
      v = log1p(t[e] + sigma * h[e]);
    } else {
      constexpr int U = 4;
      double acc = 0.0;
      for (int j0 = 0; j0 < p; j0 += U) {
        double hj[U], tj[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (j0 + u < p) {
            hj[u] = __ldcs(h + (size_t)(j0 + u) * N + e);
            if (OBJ == 0) tj[u] = __ldcs(t + (size_t)(j0 + u) * N + e);
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (j0 + u < p) {
            const int j = j0 + u;
            if (OBJ == 2) acc += __ldg(om + j) * hj[u];
            else acc += __ldg(om + j) * hj[u] / (1.0 + tj[u] + (sigma + __ldg(tau + j)) * hj[u]);
          }
      }
      v = acc;
    }
    score[e] = v;
    if (!live[e]) v = -INFINITY;
    if (better(v, e, mine.s, mine.i)) mine = Cand{v, e};
  }
  const Cand w = block_best(mine, sh);
  if (threadIdx.x == 0) best[blockIdx.x] = w;
}

// Order of the merge as integers: key of a score, larger for a better one (0: no candidate; the
// two zeros alike), then the lower index.
struct Ranked {
  unsigned long long key;
  unsigned idx;
};
POLAR_D unsigned long long score_key(double s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(s + 0.0);
  return (b >> 63) ? ~b : b | (1ull << 63);
}
POLAR_D double key_score(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k ^ (1ull << 63) : ~k));
}

POLAR_D Ranked warp_first(const Ranked& r) {
  const unsigned hi = (unsigned)(r.key >> 32), lo = (unsigned)r.key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const bool top = hi == mh && lo == ml;
  return Ranked{((unsigned long long)mh << 32) | ml, __reduce_min_sync(0xffffffffu, top ? r.idx : 0xffffffffu)};
}

// First of the block, in every thread, with one barrier: the warps' firsts go through `sh`
// (two halves used in turn) and every warp reduces them.
POLAR_D Ranked block_first(const Ranked& r, Ranked (*sh)[32], int turn) {
  const Ranked w = warp_first(r);
  if ((threadIdx.x & 31) == 0) sh[turn & 1][threadIdx.x >> 5] = w;
  __syncthreads();
  return warp_first(sh[turn & 1][threadIdx.x & 31]);
}

// The B best (one CTA).  An element among them lies in a scoring CTA whose own best is among
// the B best of the CTAs' (otherwise B elements would be better than it), so those CTAs are
// picked first and only their candidates compared.  2 B rounds of one block reduction each;
// comparing (score, index) pairs by shuffles made a round 1.6 us.
__global__ void __launch_bounds__(kMergeBlock) merge_topb_kernel(Cand* best, int nb, const double* score,
                                                                 const uint8_t* live, int N, int B, int64_t* out_idx,
                                                                 double* out_score) {
  static_assert(kMergeBlock == 1024, "one shared entry per warp");
  __shared__ Ranked sh[2][32];
  __shared__ int sel[kMaxB];
  const int tid = threadIdx.x;
  auto before = [](const Ranked& a, const Ranked& b) { return a.key > b.key || (a.key == b.key && a.idx < b.idx); };
  auto scan = [&]() {  // this thread's best CTA that is not taken
    Ranked m{0, 0xffffffffu};
    for (int i = tid; i < nb; i += kMergeBlock) {
      const Cand c = best[i];
      const Ranked r{c.i != LLONG_MAX ? score_key(c.s) : 0, (unsigned)c.i};
      if (r.key && before(r, m)) m = r;
    }
    return m;
  };
  Ranked mine = scan();
  int nsel = 0;
  for (; nsel < B && nsel < nb; ++nsel) {
    const Ranked w = block_first(mine, sh, nsel);
    if (!w.key) break;
    const int b = (int)(w.idx / kTopBlock);
    if (tid == 0) sel[nsel] = b;
    if (b % kMergeBlock == tid) {  // taken
      best[b].i = LLONG_MAX;
      mine = scan();
    }
  }
  __syncthreads();
  // candidates of this thread: position tid % kTopBlock of the CTAs tid / kTopBlock, + 4, ...
  constexpr int W = kMergeBlock / kTopBlock;
  constexpr int L = kMaxB / W;
  Ranked cd[L];  // key 0: none, or taken
#pragma unroll
  for (int k = 0; k < L; ++k) {
    cd[k] = Ranked{0, 0xffffffffu};
    if (tid / kTopBlock + W * k < nsel) {
      const long long i = (long long)sel[tid / kTopBlock + W * k] * kTopBlock + tid % kTopBlock;
      if (i < N) {
        const double v = live[i] ? score[i] : -INFINITY;
        if (!isnan(v)) cd[k] = Ranked{score_key(v), (unsigned)i};
      }
    }
  }
  auto pick = [&]() {
    Ranked m{0, 0xffffffffu};
#pragma unroll
    for (int k = 0; k < L; ++k)
      if (cd[k].key && before(cd[k], m)) m = cd[k];
    return m;
  };
  mine = pick();
  for (int b = 0; b < B; ++b) {
    const Ranked w = block_first(mine, sh, b);
    if (tid == 0) {
      out_idx[b] = w.key ? (int64_t)w.idx : LLONG_MAX;
      if (out_score) out_score[b] = w.key ? key_score(w.key) : -INFINITY;
    }
    if (w.key && mine.idx == w.idx && mine.key == w.key) {
#pragma unroll
      for (int k = 0; k < L; ++k)
        if (cd[k].idx == w.idx) cd[k].key = 0;
      mine = pick();
    }
  }
}

// ---------------------------------------------------------------------------------------
// gq[c] = sum_j om_j hh[j][c] / (1 + U[j][ia[c]][c] - U[j][ib[c]][c])   (obj 0)
//       = log1p(U[0][ia[c]][c] - U[0][ib[c]][c])                          (obj 1)
__global__ void rerank_kernel(const void* U, int u_f32, int p, int nA, int ldu, const int32_t* ia,
                              const int32_t* ib, int Br, const double* hh, const double* om, int obj, double* gq,
                              int32_t* best) {
  __shared__ double sg[1024];
  for (int c = threadIdx.x; c < Br; c += blockDim.x) {
    double g;
    if (obj == 1) {
      const double bu = ldv(U, u_f32, (size_t)ia[c] * ldu + c) - ldv(U, u_f32, (size_t)ib[c] * ldu + c);
      g = log1p(bu);
    } else {
      g = 0.0;
      for (int j = 0; j < p; ++j) {
        const double bu = ldv(U, u_f32, ((size_t)j * nA + ia[c]) * ldu + c) -
                          ldv(U, u_f32, ((size_t)j * nA + ib[c]) * ldu + c);
        g += om[j] * hh[(size_t)j * Br + c] / (1.0 + bu);
      }
    }
    gq[c] = g;
    if (c < 1024) sg[c] = g;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int bi = 0;
    double bv = sg[0];
    for (int c = 1; c < Br && c < 1024; ++c)
      if (sg[c] > bv || (isnan(sg[c]) && !isnan(bv))) {
        bv = sg[c];
        bi = c;
      }
    *best = bi;
  }
}

// ---------------------------------------------------------------------------------------
// Maintenance (polar_gpu.py:242-249).
// Row record of the maintenance: what the caches need of one (pole, active row), one sector.
struct __align__(32) MaintRow {
  double wx, wy, u, pad;
};
struct MaintTmp {
  double *xi, *eta, *D, *nxi, *neta;
  MaintRow* row;
};


static MaintTmp maint_tmp(void* base, int p, int nA, int q) {
  char* b = (char*)(((uintptr_t)base + 31) & ~uintptr_t(31));
  MaintTmp m;
  size_t o = 0;
  m.xi = (double*)(b + o); o += al256((size_t)p * q * 8);
  m.eta = (double*)(b + o); o += al256((size_t)p * q * 8);
  m.D = (double*)(b + o); o += al256((size_t)p * 8);
  m.nxi = (double*)(b + o); o += al256((size_t)p * 8);
  m.neta = (double*)(b + o); o += al256((size_t)p * 8);
  m.row = (MaintRow*)(b + o);
  return m;
}

static size_t maint_tmp_bytes(int p, int nA, int q) {
  return al256((size_t)p * q * 8) * 2 + al256((size_t)p * 8) * 3 + al256((size_t)p * nA * sizeof(MaintRow)) + 32;
}

// one CTA per pole
__global__ void maint_setup_kernel(const void* X, int ldx, const void* Y, int ldy, int f32, int p, int nA, int q,
                                   const void* U, int u_f32, int ldu, const int32_t* win, const double* G,
                                   MaintTmp m) {
  const int j = blockIdx.x;
  const int uc = win[0], a = win[1], b = win[2];
  const int64_t e = *reinterpret_cast<const int64_t*>(win + 4);
  const double* gce = G + (size_t)e * q;
  __shared__ double s1[256], s2[256];
  double n1 = 0.0, n2 = 0.0;
  for (int c = threadIdx.x; c < q; c += blockDim.x) {
    const double xi = ldv(X, f32, ((size_t)j * nA + a) * ldx + c) - ldv(X, f32, ((size_t)j * nA + b) * ldx + c);
    const double eta = gce[c] - (ldv(Y, f32, ((size_t)j * nA + a) * ldy + c) - ldv(Y, f32, ((size_t)j * nA + b) * ldy + c));
    m.xi[(size_t)j * q + c] = xi;
    m.eta[(size_t)j * q + c] = eta;
    n1 += xi * xi;
    n2 += eta * eta;
  }
  s1[threadIdx.x] = n1;
  s2[threadIdx.x] = n2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t1 = 0.0, t2 = 0.0;
    for (int i = 0; i < (int)blockDim.x; ++i) {
      t1 += s1[i];
      t2 += s2[i];
    }
    m.nxi[j] = t1;
    m.neta[j] = t2;
    m.D[j] = 1.0 + ldv(U, u_f32, ((size_t)j * nA + a) * ldu + uc) - ldv(U, u_f32, ((size_t)j * nA + b) * ldu + uc);
  }
}

// w = row . dir (before the update), then X_row -= u xi / D, Y_row += u eta / D, for the rows of
// one pole: 8 lanes per row, each with NT x VEC of its columns, whose xi and eta
// stay in registers over the CTA's rows (reading them again for every row was 2 KB from L1 for
// the row's own 512 bytes: 2,210 us at 24 x 226,000 rows, q = 64 mixed; 1,050 us now, the
// bytes of X and Y being 850).
constexpr int kMaintBlock = 256;
constexpr int kMaintRows = 512;  // rows per CTA: CTAs of pole 0, then of pole 1, ... (poles are not bounded)

template <typename T, int VEC, int NT>
__global__ void __launch_bounds__(kMaintBlock, NT <= 2 ? 3 : 1) maint_rows_kernel(T* X, int ldx, T* Y, int ldy, int nA, int q, int c0,
                                                                 int c1, const void* U, int u_f32, int ldu,
                                                                 const int32_t* win, MaintTmp m) {
  // columns [c0, c1) of q (a wide bank goes in several launches, whose dots add up)
  constexpr int LPR = 8;
  const int nb = (nA + kMaintRows - 1) / kMaintRows;
  const int j = blockIdx.x / nb, lg = threadIdx.x & (LPR - 1);
  const int uc = win[0];
  const double D = m.D[j];
  double xi[NT][VEC], eta[NT][VEC];
#pragma unroll
  for (int k = 0; k < NT; ++k)
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      const int c = c0 + (k * LPR + lg) * VEC + v;
      xi[k][v] = c < c1 ? m.xi[(size_t)j * q + c] : 0.0;
      eta[k][v] = c < c1 ? m.eta[(size_t)j * q + c] : 0.0;
    }
  const int first = (blockIdx.x - j * nb) * kMaintRows, a1 = min(nA, first + kMaintRows);
  for (int a0 = first; a0 < a1; a0 += kMaintBlock / LPR) {
    const int a = a0 + threadIdx.x / LPR;
    const bool ok = a < a1;
    T xv[NT][VEC], yv[NT][VEC];
    double u = 0.0, wx = 0.0, wy = 0.0;
    T* const xr = X + ((size_t)j * nA + a) * ldx;
    T* const yr = Y + ((size_t)j * nA + a) * ldy;
    if (ok) {
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        const int c = c0 + (k * LPR + lg) * VEC;
        if (c < c1) {
          vload<T, VEC>(xv[k], xr + c);
          vload<T, VEC>(yv[k], yr + c);
        }
      }
      u = ldv(U, u_f32, ((size_t)j * nA + a) * ldu + uc);
      const double ud = u / D;
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        const int c = c0 + (k * LPR + lg) * VEC;
        if (c < c1) {
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const double x = (double)xv[k][v], y = (double)yv[k][v];
            wx = fma(x, xi[k][v], wx);
            wy = fma(y, eta[k][v], wy);
            xv[k][v] = (T)fma(-ud, xi[k][v], x);
            yv[k][v] = (T)fma(ud, eta[k][v], y);
          }
          vstore<T, VEC>(xr + c, xv[k]);
          vstore<T, VEC>(yr + c, yv[k]);
        }
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      wx += __shfl_xor_sync(0xffffffffu, wx, o);
      wy += __shfl_xor_sync(0xffffffffu, wy, o);
    }
    if (ok && lg == 0) {
      MaintRow& r = m.row[(size_t)j * nA + a];
      if (c0 > 0) {
        wx += r.wx;
        wy += r.wy;
      }
      r = MaintRow{wx, wy, u, 0.0};
    }
  }
}

// Cache change of item (pole j, candidate e): its two row records are one sector each.
POLAR_D void maint_change(const MaintTmp& m, const int32_t* es, int nA, int j, int e, double& dh, double& dt) {
  const MaintRow ra = m.row[(size_t)j * nA + es[2 * (size_t)e]], rb = m.row[(size_t)j * nA + es[2 * (size_t)e + 1]];
  const double cc = (ra.u - rb.u) / m.D[j];
  dh = cc * cc * m.nxi[j] - 2.0 * cc * (ra.wx - rb.wx);
  dt = cc * cc * m.neta[j] + 2.0 * cc * (ra.wy - rb.wy);
}

__global__ void maint_cache_kernel(int p, int nA, int N, const int32_t* es, MaintTmp m, double* h, double* t) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)p * N) return;
  const int j = (int)(g / N), e = (int)(g % N);
  double dh, dt;
  maint_change(m, es, nA, j, e, dh, dt);
  h[g] = fmax(0.0, h[g] + dh);
  t[g] = fmax(0.0, t[g] + dt);
}

// Column-split form (the sketch columns spread over several ranks): this rank's share of
// the cache change, summed over the ranks before cache_apply_kernel clamps it in.
__global__ void maint_delta_kernel(int p, int nA, int N, const int32_t* es, MaintTmp m, double* dh, double* dt) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)p * N) return;
  const int j = (int)(g / N), e = (int)(g % N);
  maint_change(m, es, nA, j, e, dh[g], dt[g]);
}

__global__ void cache_apply_kernel(double* h, const double* dh, double* t, const double* dt, long long count) {
  for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < count; o += (long long)gridDim.x * blockDim.x) {
    h[o] = fmax(0.0, h[o] + dh[o]);
    t[o] = fmax(0.0, t[o] + dt[o]);
  }
}

// Winner record: win[0] = shortlist position, win[1] = aa, win[2] = bb, win[4..5] = e.
__global__ void select_kernel(const int64_t* shortl, const int32_t* best, const int32_t* es, uint8_t* live,
                              int32_t* win) {
  if (threadIdx.x != 0) return;
  const int b = best ? *best : 0;
  const int64_t e = shortl[b];
  win[0] = b;
  win[1] = es[2 * e];
  win[2] = es[2 * e + 1];
  win[3] = 0;
  *reinterpret_cast<int64_t*>(win + 4) = e;
  if (live) live[e] = 0;
}

__global__ void rank1_rows_kernel(double* F, int ldf, int q, const double* G, const int64_t* cand, const int64_t* sel) {
  const int64_t e = *sel;  // sel may point at win[4..5]
  const int64_t a = cand[2 * e], b = cand[2 * e + 1];
  for (int c = threadIdx.x; c < q; c += blockDim.x) {
    const double g = G[(size_t)e * q + c];
    F[(size_t)a * ldf + c] += g;
    F[(size_t)b * ldf + c] -= g;
  }
}

static int check_launch(const char* what) {
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_cuda_error(what, e);
  return POLAR_OK;
}

}  // namespace polar

using namespace polar;

extern "C" int polar_fill_incidence(int n, int R, const int64_t* d_cand, const int64_t* d_sel, const int32_t* d_es,
                                    double* d_W, int ldw, int32_t* d_ia, int32_t* d_ib, polar_stream_t stream) {
  clear_error();
  if (n < 1 || R < 1 || ldw < R || !d_cand || !d_sel || !d_W) return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  if ((d_ia || d_ib) && !d_es) return set_error(POLAR_ERR_BAD_ARG, "ia/ib need es");
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(d_W, 0, sizeof(double) * (size_t)n * ldw, st);
  if (e != cudaSuccess) return set_cuda_error("cudaMemsetAsync", e);
  fill_incidence_kernel<<<(R + 127) / 128, 128, 0, st>>>(R, d_cand, d_sel, d_es, d_W, ldw, d_ia, d_ib);
  return check_launch("fill_incidence");
}

extern "C" int polar_pair_norms(const void* d_X, int x_f32, int p, int nA, int ldx, int col0, int q,
                                const int32_t* d_ea, const int32_t* d_eb, int N, double* d_out, polar_stream_t stream) {
  clear_error();
  if (!d_X || !d_ea || !d_eb || !d_out || p < 1 || nA < 1 || q < 1 || N < 0 || col0 + q > ldx)
    return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  if (N == 0) return POLAR_OK;
  const long long threads = (long long)p * N * 16;
  const int blocks = (int)((threads + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  if (x_f32)
    pair_norms_kernel<float><<<blocks, 256, 0, st>>>((const float*)d_X, p, nA, ldx, col0, q, d_ea, d_eb, N, d_out);
  else
    pair_norms_kernel<double><<<blocks, 256, 0, st>>>((const double*)d_X, p, nA, ldx, col0, q, d_ea, d_eb, N, d_out);
  return check_launch("pair_norms");
}

extern "C" size_t polar_topb_tmp_bytes(int N, int B) {
  (void)B;
  const size_t n = N > 0 ? N : 1;
  return al256(n * sizeof(double)) + (n + kTopBlock - 1) / kTopBlock * sizeof(Cand) + 256;
}

extern "C" int polar_score_topb(const double* d_h, const double* d_t, const double* d_tau, const double* d_om,
                                double sigma, int p, int N, const uint8_t* d_live, int obj, int B, int64_t* d_out_idx,
                                double* d_out_score, double* d_score_all, void* d_tmp, polar_stream_t stream) {
  clear_error();
  if (!d_h || !d_t || !d_tau || !d_om || !d_live || !d_out_idx || !d_tmp || p < 1 || N < 1)
    return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  if (B < 1 || B > kMaxB || B > N) return set_error(POLAR_ERR_BAD_ARG, "B out of range");
  if (obj < 0 || obj > 2) return set_error(POLAR_ERR_BAD_ARG, "obj must be 0, 1 or 2");
  const int nb = (int)(((long long)N + kTopBlock - 1) / kTopBlock);
  cudaStream_t st = (cudaStream_t)stream;
  double* score = d_score_all ? d_score_all : (double*)d_tmp;
  Cand* best = (Cand*)((char*)d_tmp + al256((size_t)N * sizeof(double)));
  auto* k = obj == 1 ? score_kernel<1> : obj == 2 ? score_kernel<2> : score_kernel<0>;
  k<<<nb, kTopBlock, 0, st>>>(d_h, d_t, d_tau, d_om, sigma, p, N, d_live, score, best);
  const int rc = check_launch("score");
  if (rc) return rc;
  merge_topb_kernel<<<1, kMergeBlock, 0, st>>>(best, nb, score, d_live, N, B, d_out_idx, d_out_score);
  return check_launch("merge_topb");
}

extern "C" int polar_rerank(const void* d_U, int u_f32, int p, int nA, int ldu, const int32_t* d_ia,
                            const int32_t* d_ib, int Br, const double* d_hh, const double* d_om, int obj, double* d_gq,
                            int32_t* d_best, polar_stream_t stream) {
  clear_error();
  if (!d_U || !d_ia || !d_ib || !d_gq || !d_best || Br < 1 || Br > 1024 || ldu < Br || p < 1)
    return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  if (obj == 0 && (!d_hh || !d_om)) return set_error(POLAR_ERR_BAD_ARG, "frac re-rank needs hh and om");
  rerank_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(d_U, u_f32, p, nA, ldu, d_ia, d_ib, Br, d_hh, d_om, obj, d_gq,
                                                     d_best);
  return check_launch("rerank");
}

extern "C" size_t polar_maintain_tmp_bytes(int p, int nA, int q) { return maint_tmp_bytes(p, nA, q); }

extern "C" int polar_select(const int64_t* d_short, const int32_t* d_best, const int32_t* d_es, uint8_t* d_live,
                            int32_t* d_win, polar_stream_t stream) {
  clear_error();
  if (!d_short || !d_es || !d_win) return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  select_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(d_short, d_best, d_es, d_live, d_win);
  return check_launch("select");
}

// Both maintenance forms: delta == false updates h, t in place; delta == true writes this
// rank's cache change to h, t (as dh, dt).
static int maintain(void* d_X, int ldx, void* d_Y, int ldy, int xy_f32, int p, int nA, int q, const void* d_U,
                    int u_f32, int ldu, const int32_t* d_win, const double* d_G, const int32_t* d_es, int N,
                    double* d_h, double* d_t, void* d_tmp, polar_stream_t stream, bool delta) {
  clear_error();
  if (!d_X || !d_Y || !d_U || !d_win || !d_G || !d_es || !d_h || !d_t || !d_tmp || p < 1 || nA < 1 || q < 1 ||
      ldx < q || ldy < q)
    return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  MaintTmp m = maint_tmp(d_tmp, p, nA, q);
  maint_setup_kernel<<<p, 128, 0, st>>>(d_X, ldx, d_Y, ldy, xy_f32, p, nA, q, d_U, u_f32, ldu, d_win, d_G, m);
  int rc = check_launch("maint_setup");
  if (rc) return rc;
  const uintptr_t al = (uintptr_t)d_X | (uintptr_t)d_Y;
  const int ctas = (nA + kMaintRows - 1) / kMaintRows * p;
  auto rows = [&](auto* x, auto* y, auto vec) {
    using T = std::remove_pointer_t<decltype(x)>;
    constexpr int V = decltype(vec)::value;
    for (int c0 = 0; c0 < q; c0 += 8 * 8 * V) {
      const int c1 = q - c0 < 8 * 8 * V ? q : c0 + 8 * 8 * V;
      const int trips = (c1 - c0 + 8 * V - 1) / (8 * V);
      auto go = [&](auto nt) {
        maint_rows_kernel<T, V, decltype(nt)::value><<<ctas, kMaintBlock, 0, st>>>(x, ldx, y, ldy, nA, q, c0, c1, d_U,
                                                                                   u_f32, ldu, d_win, m);
      };
      if (trips <= 1) go(std::integral_constant<int, 1>{});
      else if (trips <= 2) go(std::integral_constant<int, 2>{});
      else if (trips <= 4) go(std::integral_constant<int, 4>{});
      else go(std::integral_constant<int, 8>{});
    }
  };
  if (xy_f32) {
    if (q % 4 == 0 && ldx % 4 == 0 && ldy % 4 == 0 && al % 16 == 0)
      rows((float*)d_X, (float*)d_Y, std::integral_constant<int, 4>{});
    else
      rows((float*)d_X, (float*)d_Y, std::integral_constant<int, 1>{});
  } else {
    if (q % 2 == 0 && ldx % 2 == 0 && ldy % 2 == 0 && al % 16 == 0)
      rows((double*)d_X, (double*)d_Y, std::integral_constant<int, 2>{});
    else
      rows((double*)d_X, (double*)d_Y, std::integral_constant<int, 1>{});
  }
  rc = check_launch("maint_rows");
  if (rc) return rc;
  if (N > 0) {
    const long long t2 = (long long)p * N;
    if (delta)
      maint_delta_kernel<<<(int)((t2 + 255) / 256), 256, 0, st>>>(p, nA, N, d_es, m, d_h, d_t);
    else
      maint_cache_kernel<<<(int)((t2 + 255) / 256), 256, 0, st>>>(p, nA, N, d_es, m, d_h, d_t);
    rc = check_launch(delta ? "maint_delta" : "maint_cache");
  }
  return rc;
}

extern "C" int polar_maintain(void* d_X, int ldx, void* d_Y, int ldy, int xy_f32, int p, int nA, int q, const void* d_U,
                              int u_f32, int ldu, const int32_t* d_win, const double* d_G, const int32_t* d_es, int N,
                              double* d_h, double* d_t, void* d_tmp, polar_stream_t stream) {
  return maintain(d_X, ldx, d_Y, ldy, xy_f32, p, nA, q, d_U, u_f32, ldu, d_win, d_G, d_es, N, d_h, d_t, d_tmp, stream,
                  false);
}

extern "C" int polar_maintain_split(void* d_X, int ldx, void* d_Y, int ldy, int xy_f32, int p, int nA, int q,
                                    const void* d_U, int u_f32, int ldu, const int32_t* d_win, const double* d_G,
                                    const int32_t* d_es, int N, double* d_dh, double* d_dt, void* d_tmp,
                                    polar_stream_t stream) {
  return maintain(d_X, ldx, d_Y, ldy, xy_f32, p, nA, q, d_U, u_f32, ldu, d_win, d_G, d_es, N, d_dh, d_dt, d_tmp,
                  stream, true);
}

extern "C" int polar_cache_apply(double* d_h, const double* d_dh, double* d_t, const double* d_dt, int64_t count,
                                 polar_stream_t stream) {
  clear_error();
  if (!d_h || !d_dh || !d_t || !d_dt || count < 0) return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  if (count == 0) return POLAR_OK;
  const long long blocks = (count + 255) / 256;
  cache_apply_kernel<<<(int)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(d_h, d_dh, d_t,
                                                                                                     d_dt, count);
  return check_launch("cache_apply");
}

extern "C" int polar_rank1_rows(double* d_F, int ldf, int q, const double* d_G, const int64_t* d_cand,
                                const int64_t* d_sel, polar_stream_t stream) {
  clear_error();
  if (!d_F || !d_G || !d_cand || !d_sel || q < 1 || ldf < q) return set_error(POLAR_ERR_BAD_ARG, "bad arguments");
  rank1_rows_kernel<<<1, 128, 0, (cudaStream_t)stream>>>(d_F, ldf, q, d_G, d_cand, d_sel);
  return check_launch("rank1_rows");
}
