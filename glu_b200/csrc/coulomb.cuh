// Coulomb gauge fixing of every time slice at once (GLU's Coulomb_FA,
// src/Gfix/CFACG.c:531-636, solves the slices one after the other; they are
// independent problems on the original spatial links, so here all of them
// advance together, each with its own scalars, iteration count and end).
//
// Per slice t the unknown is the slice gauge field g_t(x) (SoA [9][V], the
// slices side by side), the derivative is taken on the rotated links
// g(x) U_i(x,t) g(x+i)^dag (steep_deriv_CG, CFACG.c:91-163), the FFT is the
// 3D transform of each slice (FOURIER_ACCELERATE2) done by the Landau passes
// with ndim = 3, and the update is g <- reunit(1 + a A) g
// (exponentiate_gauge_CG, line_search.c:101-115).  Each step of a slice is
// either an SD step (a run's first step, every FASD step) or a CG step.
// A slice whose run ends is reunitarised and checked (adequate_solution,
// CFACG.c:432-456), continued, or restarted from a random g (steep_fix,
// CFACG.c:459-529); finished slices are masked out of every kernel.
#pragma once

#include "kernels.cuh"

namespace gfix {

template <typename R>
struct CCtx {
  cx<R> *U;           // links SoA [4][9][V]
  cx<R> *g;           // slice gauge fields SoA [9][V]
  cx<R> *fb[2];       // in / in_old
  cx<R> *sb[2];       // sn ping-pong
  DevState *st;       // parities (shared with the FFT passes)
  CoulState *cs;
  Slice *sl;
  double *part;       // [nslices][nbs][2]
  unsigned *tick;     // a ticket for each slice, zero between kernels
  int L[4];
  int V, Lcu, nbs;
};

// slice-site coordinates and the in-slice neighbours of site i in direction
// MU (compile-time, so no index array lands in local memory)
struct SliceSite {
  int i, x[3];
};
__device__ __forceinline__ SliceSite slice_site(int i, const int *L) {
  SliceSite q;
  q.i = i;
  q.x[0] = i % L[0];
  const int r = i / L[0];
  q.x[1] = r % L[1];
  q.x[2] = r / L[1];
  return q;
}
template <int MU>
__device__ __forceinline__ int sfwd(const SliceSite &q, const int *L) {
  const int sd = MU == 0 ? 1 : MU == 1 ? L[0] : L[0] * L[1];
  return q.x[MU] == L[MU] - 1 ? q.i - (L[MU] - 1) * sd : q.i + sd;
}
// the same with a run-time direction, by selects
__device__ __forceinline__ int sfwd_rt(const SliceSite &q, const int *L, int mu) {
  const int xm = mu == 0 ? q.x[0] : mu == 1 ? q.x[1] : q.x[2];
  const int lm = mu == 0 ? L[0] : mu == 1 ? L[1] : L[2];
  const int sd = mu == 0 ? 1 : mu == 1 ? L[0] : L[0] * L[1];
  return xm == lm - 1 ? q.i - (lm - 1) * sd : q.i + sd;
}
template <int MU>
__device__ __forceinline__ int sbck(const SliceSite &q, const int *L) {
  const int sd = MU == 0 ? 1 : MU == 1 ? L[0] : L[0] * L[1];
  return q.x[MU] == 0 ? q.i + (L[MU] - 1) * sd : q.i - sd;
}

template <typename R>
__device__ __forceinline__ void load9(const cx<R> *p, int V, int s, cx<R> *u) {
#pragma unroll
  for (int e = 0; e < 9; e++) u[e] = p[(size_t)e * V + s];
}
template <typename R>
__device__ __forceinline__ void store9(cx<R> *p, int V, int s, const cx<R> *u) {
#pragma unroll
  for (int e = 0; e < 9; e++) p[(size_t)e * V + s] = u[e];
}

template <typename CT, typename R>
__device__ __forceinline__ cx<CT> up_to(cx<R> a) {
  return mk<CT>((CT)a.x, (CT)a.y);
}

// ---------------------------------------------------------------------
// derivative on the rotated links W_i(x) = g(x) U_i(x) g(x+i)^dag, packed like
// the Landau fields (steep_deriv_CG, src/Gfix/CFACG.c:91-163): the traceless
// anti-Hermitian part of sum_i W_i(x-i) - W_i(x).
//
// In FP64 arithmetic the links are not formed.  W and -W^dag have the same
// part, so with
//   S(x) = sum_i U_i(x) g(x+i)^dag + (g(x-i) U_i(x-i))^dag
// it is that of -g(x) S(x): one product for each of the six links and one
// with g(x), in place of two for each.  Every column of a product is formed
// from those of its factors: a third column completed from the first two would
// differ, for a g off SU(3) (FP32 storage, or the drift of a long run), from
// what the neighbour's sum holds of the same link, and the two would no longer
// cancel in the sum over the slice, which turns the slice as a whole.  A
// product's three terms are added before they meet the sum.  Rms error of a
// site against 128 bits: 0.5 to 0.85 of that of six links formed by two products
// each.  32^3 x 64: 0.326 -> 0.239 ms (four blocks per SM).
//
// FP32 arithmetic (FP32 storage, theta >= hp_below) forms the links: the same
// bits at both ends of each, whose sum over the slice cancels to the last,
// where the rounding of -g S in 32 bits turned the slice, and a mixed fix ended
// 1.1 to 1.4 times as far from the same in 64 bits (0.16 instead of 0.23 ms).
template <typename R, typename CT>
__device__ __forceinline__ void link_ct(const CCtx<R> &c, int mu, int s, cx<CT> *U) {
  cx<R> t[9];
  load_link(c.U, c.V, mu, s, t);
#pragma unroll
  for (int e = 0; e < 9; e++) U[e] = up_to<CT>(t[e]);
  if constexpr (sizeof(CT) != sizeof(R)) complete_col2(U);
}
template <typename R, typename CT>
__device__ __forceinline__ void gauge_ct(const CCtx<R> &c, int s, cx<CT> *G) {
#pragma unroll
  for (int e = 0; e < 9; e++) G[e] = up_to<CT>(c.g[(size_t)e * c.V + s]);
}
// a b + s of row-times-column triples, the three terms first
template <typename CT>
__device__ __forceinline__ cx<CT> add_dot(cx<CT> s, cx<CT> a0, cx<CT> b0, cx<CT> a1, cx<CT> b1,
                                          cx<CT> a2, cx<CT> b2) {
  return cadd(s, cmadd(cmadd(cmul(a0, b0), a1, b1), a2, b2));
}

// S += U_MU(x) g(x+MU)^dag + (g(x-MU) U_MU(x-MU))^dag
template <typename R, typename CT, int MU>
__device__ __forceinline__ void cderiv_dir(const CCtx<R> &c, const SliceSite &q,
                                           int off, cx<CT> *S) {
  const int it = off + sfwd<MU>(q, c.L), bk = off + sbck<MU>(q, c.L);
  cx<CT> U[9], G[9];
  link_ct(c, MU, off + q.i, U);
  gauge_ct(c, it, G);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      S[3 * i + j] = add_dot(S[3 * i + j], U[3 * i], conjg(G[3 * j]), U[3 * i + 1],
                             conjg(G[3 * j + 1]), U[3 * i + 2], conjg(G[3 * j + 2]));
  link_ct(c, MU, bk, U);
  gauge_ct(c, bk, G);
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int r = 0; r < 3; r++)
      S[3 * k + r] = add_dot(S[3 * k + r], conjg(G[3 * r]), conjg(U[k]), conjg(G[3 * r + 1]),
                             conjg(U[3 + k]), conjg(G[3 * r + 2]), conjg(U[6 + k]));
}

// Hermitian short form of a matrix (herm_short)
template <typename CT>
struct HShort {
  CT h0, h3;
  cx<CT> h1, h2, h4;
};
// that of the link g(a) U_MU(a) g(b)^dag
template <typename R, typename CT>
__device__ __forceinline__ HShort<CT> rotated_herm(const CCtx<R> &c, int mu, int a, int b) {
  cx<CT> C[9], A[9], B[9];
  link_ct(c, mu, a, C);
  gauge_ct(c, a, A);
  gauge_ct(c, b, B);
  gtransform(A, C, B);
  HShort<CT> h;
  herm_short(C, h.h0, h.h1, h.h2, h.h3, h.h4);
  return h;
}
// H += that of W_MU(x-MU), less that of W_MU(x)
template <typename R, typename CT, int MU>
__device__ __forceinline__ void cderiv_links(const CCtx<R> &c, const SliceSite &q, int off,
                                             HShort<CT> &H) {
  const int x = off + q.i, it = off + sfwd<MU>(q, c.L), bk = off + sbck<MU>(q, c.L);
  const HShort<CT> b = rotated_herm<R, CT>(c, MU, x, it);
  const HShort<CT> a = rotated_herm<R, CT>(c, MU, bk, x);
  H.h0 += a.h0 - b.h0;
  H.h1 = cadd(H.h1, csub(a.h1, b.h1));
  H.h2 = cadd(H.h2, csub(a.h2, b.h2));
  H.h3 += a.h3 - b.h3;
  H.h4 = cadd(H.h4, csub(a.h4, b.h4));
}

// CT: arithmetic type.  With FP32 storage a slice below theta = hp_below is
// worked in FP64 arithmetic: the rotated links g U g^dag of FP32 products
// carry a per-step rounding noise that stalls the FP32 phase near
// theta ~ 1e-8.  `sel` picks the slices of this variant (ArithSel).
template <typename R, typename CT = R>
__global__ void __launch_bounds__(kCoulThreads, 4) k_cderiv(CCtx<R> c, int sel) {
  const int t = blockIdx.y;
  if (c.sl[t].mode == SL_DONE || arith_skip(sel, c.sl[t].tr, c.cs->hp_below))
    return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // in-slice site
  if (i >= c.Lcu) return;
  const SliceSite q = slice_site(i, c.L);
  const int off = t * c.Lcu;
  HShort<CT> H;  // the sum's Hermitian short form
  if constexpr (sizeof(CT) == 4) {
    H.h0 = H.h3 = 0;
    H.h1 = H.h2 = H.h4 = mk<CT>(0, 0);
    cderiv_links<R, CT, 0>(c, q, off, H);
    cderiv_links<R, CT, 1>(c, q, off, H);
    cderiv_links<R, CT, 2>(c, q, off, H);
  } else {
    cx<CT> S[9], G[9], M[9];
#pragma unroll
    for (int e = 0; e < 9; e++) S[e] = mk<CT>(0, 0);
    cderiv_dir<R, CT, 0>(c, q, off, S);
    cderiv_dir<R, CT, 1>(c, q, off, S);
    cderiv_dir<R, CT, 2>(c, q, off, S);
    gauge_ct(c, off + i, G);
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const cx<CT> m = cmadd(cmadd(cmul(G[3 * r], S[k]), G[3 * r + 1], S[3 + k]),
                               G[3 * r + 2], S[6 + k]);
        M[3 * r + k] = mk<CT>(-m.x, -m.y);
      }
    herm_short(M, H.h0, H.h1, H.h2, H.h3, H.h4);
  }
  // pack: in0 = i Re s0 - Re s3, in_k = i Re s_k - Im s_k (CFACG.c:144-150)
  cx<R> *f = pick(c.fb, c.st->parity);
  const size_t V = c.V, s = off + i;
  f[s] = mk<R>((R)-H.h3, (R)H.h0);
  f[V + s] = mk<R>((R)-H.h1.y, (R)H.h1.x);
  f[2 * V + s] = mk<R>((R)-H.h2.y, (R)H.h2.x);
  f[3 * V + s] = mk<R>((R)-H.h4.y, (R)H.h4.x);
}

// The sums of the accelerated field, insum (sum_DER2 / sum_PR, one norm) and
// sum_conj (src/Gfix/CFACG.c:165-258), come from the inverse xy FFT pass
// (prsum = 1): its per-plane partials of slice t are the planes
// t Lz .. t Lz + Lz - 1 of each of the 4 fields.

// sn = in + beta sn_old at site s (the same fma form as the Landau kernels);
// an SD step takes sn = in without reading sn_old
template <typename R>
__device__ __forceinline__ void cdir(const cx<R> *in, const cx<R> *so, R beta,
                                     bool sd, size_t s, size_t V, cx<R> *f) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const cx<R> a = in[k * V + s];
    if (sd) {
      f[k] = a;
    } else {
      const cx<R> b = so[k * V + s];
      f[k] = mk<R>(fma(beta, b.x, a.x), fma(beta, b.y, a.y));
    }
  }
}

// direction sn = in + beta_t sn_old (an SD step takes sn = in), written for
// every live slice, and the line-search probes of line_search_Coulomb
// (src/Gfix/line_search.c:141-271) at 0.17 and 0.34 as differences to the
// alpha = 0 value; each link counted once (the forward links of every site,
// the same set the reference's draughtboard visits).  Per link the first
// two columns of the rotated link g(x) U g(x+mu)^dag are formed once and serve
// both probes (probe_trace); the probe gauge matrices of the site itself wait
// in shared memory.  At 32^3 x 64: 0.453 -> 0.403 ms in FP64, bound by its
// arithmetic at three blocks per SM, 0.300 -> 0.269 ms in FP32 at four.
// CT: arithmetic type of the probes (FP64 for FP32 storage below hp_below,
// as in k_cderiv); `sel` picks the slices of this variant.
template <typename R, typename CT = R>
__global__ void __launch_bounds__(kCoulThreads, sizeof(CT) == 4 ? 4 : 3) k_cprobe(CCtx<R> c, int sel) {
  __shared__ cx<CT> sA[2][9][kCoulThreads];
  const int t = blockIdx.y;
  const Slice &S = c.sl[t];
  if (S.mode == SL_DONE || arith_skip(sel, S.tr, c.cs->hp_below)) return;
  double v[2] = {0.0, 0.0};
  const bool probes = S.use_ls;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.Lcu) {
    const int par = c.st->parity, spar = c.st->sparity;
    const cx<R> *in = pick(c.fb, par), *so = pick(c.sb, spar);
    cx<R> *sn = pick(c.sb, spar ^ 1);
    const R beta = (R)S.beta;
    const bool sdstep = S.sd != 0;
    const int off = t * c.Lcu;
    cx<R> f[4];
    cdir(in, so, beta, sdstep, (size_t)off + i, (size_t)c.V, f);
#pragma unroll
    for (int k = 0; k < 4; k++) sn[(size_t)k * c.V + off + i] = f[k];
    if (probes) {
      auto up = [](cx<R> a) { return mk<CT>((CT)a.x, (CT)a.y); };
      const CT al0 = CT(0.17), al1 = CT(0.34);
#pragma unroll 1
      for (int k = 0; k < 2; k++) {
        cx<CT> A[9];
        set_gauge(A, up(f[0]), up(f[1]), up(f[2]), up(f[3]), k ? al1 : al0);
#pragma unroll
        for (int e = 0; e < 9; e++) sA[k][e][threadIdx.x] = A[e];
      }
      const SliceSite q = slice_site(i, c.L);
      CT d[2] = {0, 0};
#pragma unroll 1
      for (int mu = 0; mu < 3; mu++) {
        const int it = sfwd_rt(q, c.L, mu);
        // the first two columns of C = g(x) U g(x+mu)^dag
        cx<CT> w0[3], w1[3];
        {
          cx<R> t9[9];
          cx<CT> U[9], G[9], b0[3], b1[3];
          load_link(c.U, c.V, mu, off + i, t9);
#pragma unroll
          for (int e = 0; e < 9; e++) U[e] = up(t9[e]);
          if constexpr (sizeof(CT) != sizeof(R)) complete_col2(U);
#pragma unroll
          for (int e = 0; e < 6; e++) G[e] = up(c.g[(size_t)e * c.V + off + it]);
#pragma unroll
          for (int r = 0; r < 3; r++) {
            b0[r] = cmaddc(cmaddc(cmulc(U[3 * r], G[0]), U[3 * r + 1], G[1]), U[3 * r + 2], G[2]);
            b1[r] = cmaddc(cmaddc(cmulc(U[3 * r], G[3]), U[3 * r + 1], G[4]), U[3 * r + 2], G[5]);
          }
          load9(c.g, c.V, off + i, t9);
#pragma unroll
          for (int e = 0; e < 9; e++) G[e] = up(t9[e]);
          mat_vec(w0, G, b0);
          mat_vec(w1, G, b1);
        }
        const CT t0 = re_tr_cols(w0, w1);
        cx<R> fy[4];
        cdir(in, so, beta, sdstep, (size_t)off + it, (size_t)c.V, fy);
        const ProbeDir<CT> p = probe_dir(up(fy[0]), up(fy[1]), up(fy[2]), up(fy[3]));
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
          cx<CT> A[9];
#pragma unroll
          for (int e = 0; e < 9; e++) A[e] = sA[k][e][threadIdx.x];
          d[k] += probe_trace(A, w0, w1, p, k ? al1 : al0) - t0;
        }
      }
      v[0] = d[0];
      v[1] = d[1];
    }
  }
  if (probes) block_sum_store<2>(v, c.part + 2 * ((size_t)t * c.nbs + blockIdx.x));
}

// g(x) <- reunit(1 + alpha_t sn(x)) g(x) (exponentiate_gauge_CG,
// src/Gfix/line_search.c:101-115)
template <typename R>
__global__ void __launch_bounds__(kCoulThreads) k_cupdate(CCtx<R> c) {
  // (from the last site to the first, whose g and fields the probes before it
  // left in L2: 32^3 x 64 0.126 -> 0.123 ms in FP64, 0.0585 -> 0.0556 in FP32)
  const int t = gridDim.y - 1 - blockIdx.y;
  const Slice &S = c.sl[t];
  if (S.mode == SL_DONE) return;
  const int i = (gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= c.Lcu) return;
  const size_t V = c.V, s = (size_t)t * c.Lcu + i;
  const cx<R> *d = pick(c.sb, c.st->sparity ^ 1);
  cx<R> A[9], G[9], r[9];
  set_gauge(A, d[s], d[V + s], d[2 * V + s], d[3 * V + s], (R)S.alpha);
  load9(c.g, c.V, (int)s, G);
  multab(r, A, G);
  // FP32: the product of many rounded SU(3) factors drifts off the group
  // (~1e-7 a step) and the derivative assumes a unitary g; FP64 keeps GLU's
  // plain product
  if constexpr (sizeof(R) == 4) gram_reunit(r);
  store9(c.g, c.V, (int)s, r);
}

// per-slice housekeeping at the end of a run: reunitarise g_t and check its
// norm (adequate_solution, src/Gfix/CFACG.c:432-456), or replace g_t by
// random SU(3) matrices for a restart (steep_fix, CFACG.c:507-522; our own
// generator, not GLU's RNG stream)
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// what = 0: reunitarise and check, then the end of a run of the slices that
// have ended theirs; what = 1: random restarts, and the in / in_old and sn
// ping-pong after every step.  Few slices need either in any step, so the
// grid holds kMaintBlocks blocks a slice, which loop over its sites (a block
// for every 128 sites returned at once, but cost 0.14 ms a launch at
// 64^3 x 128).
constexpr int kMaintBlocks = 8;

template <typename R>
__global__ void __launch_bounds__(kCoulThreads) k_cmaint(CCtx<R> c, int what) {
  if (c.st->done) return;
  const int t = blockIdx.y;
  Slice &S = c.sl[t];
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (what == 1 && t == 0 && i0 == 0) {
    c.st->parity ^= 1;
    c.st->sparity ^= 1;
  }
  if (S.mode == SL_DONE) return;
  if (what == 0 && S.sd == -1) {
    if (S.reunit)
      for (int i = i0; i < c.Lcu; i += step) {
        const int s = t * c.Lcu + i;
        cx<R> G[9];
        load9(c.g, c.V, s, G);
        gram_reunit(G);
        store9(c.g, c.V, s, G);
        double sum = 0.0;
#pragma unroll
        for (int e = 0; e < 9; e++) sum += (double)G[e].x * G[e].x + (double)G[e].y * G[e].y;
        const double lim = (double)(S.iter > 0 ? S.iter : 1) * c.cs->prec_tol;
        if (fabs(sum - 3.0) > lim) atomicOr(&S.bad, 1);
      }
    if (arrive_last(c.tick + t, gridDim.x) && threadIdx.x == 0)
      apply_slice(c.cs, c.sl, c.st, t, C_END2, 0.0, 0.0, (double)c.Lcu);
  } else if (what == 1 && S.randomize) {
    for (int i = i0; i < c.Lcu; i += step) {
      cx<R> G[9];
      unsigned long long h = mix64(c.cs->seed ^ mix64(((unsigned long long)t << 40) ^
                                                      ((unsigned long long)S.control << 32) ^
                                                      (unsigned long long)i));
#pragma unroll
      for (int e = 0; e < 9; e++) {
        h = mix64(h);
        const double u1 = ((h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
        h = mix64(h);
        const double u2 = ((h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
        const double rad = sqrt(-2.0 * log(u1));
        G[e] = mk<R>((R)(rad * cospi(2.0 * u2)), (R)(rad * sinpi(2.0 * u2)));
      }
      gram_reunit(G);
      store9(c.g, c.V, t * c.Lcu + i, G);
    }
  }
}

// one warp per slice: fixed-order sums of the slice's partials (each lane
// a strided subset in order, then a fixed shuffle tree), then the scalar step
// on lane 0.  Partials: C_SUMS reads the inverse xy pass's pairs (`bps` blocks
// of the slice in each field, field-major), C_PROBES the probe kernel's
// per-block pairs (t * nbs + block).  C_PROBES also ends the step (C_END1: the
// update that follows reads neither).  Tickets in those kernels in place of
// these launches cost more than they saved (probes 0.403 -> 0.442 ms at 32^3
// x 64): their grids must have a block for every 128 sites of each slice, as
// any number of slices may be left.
constexpr int kCScalarSlices = 4;  // slices (warps) per block

__global__ void __launch_bounds__(32 * kCScalarSlices)
    k_cscalar(CoulState *cs, Slice *sl, const double *part, int nbs, int bps, int op,
              double Lcu, DevState *st) {
  const int t = blockIdx.x * kCScalarSlices + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= cs->nslices || sl[t].mode == SL_DONE) return;
  const size_t np = (size_t)bps * cs->nslices;
  const int n = op == C_SUMS ? 4 * bps : nbs;
  double a0 = 0.0, a1 = 0.0;
  constexpr int kU = 4;
  for (int b0 = lane; b0 < n; b0 += 32 * kU) {
    double x0[kU], x1[kU];
#pragma unroll
    for (int k = 0; k < kU; k++) {
      const int b = b0 + 32 * k;
      const size_t i = op == C_SUMS ? (b / bps) * np + (size_t)t * bps + b % bps
                                    : (size_t)t * nbs + b;
      x0[k] = b < n ? part[2 * i] : 0.0;
      x1[k] = b < n ? part[2 * i + 1] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kU; k++) {
      a0 += x0[k];
      a1 += x1[k];
    }
  }
  a0 = warp_sum(a0);
  a1 = warp_sum(a1);
  if (lane != 0) return;
  apply_slice(cs, sl, st, t, op, a0, a1, Lcu);
  if (op == C_PROBES) apply_slice(cs, sl, st, t, C_END1, 0.0, 0.0, Lcu);
}

// the slice transforms of Coulomb_FA (gtransform_slice, src/Gfix/gtrans.c:
// 214-238): U_i(x,t) <- g_t(x) U_i(x,t) g_t(x+i)^dag for i < 3 and
// U_t(x,t) <- g_t(x) U_t(x,t) g_{t+1}(x)^dag.  ALL_T: every temporal link,
// periodic in t (a whole lattice); otherwise the last slice's temporal links
// are left for k_cfinish_aos (a block of slices whose successor slice lives
// elsewhere).
template <typename R, int MU>
__device__ __forceinline__ void cslice_link(const CCtx<R> &c, const SliceSite &q,
                                            int s, int t, const cx<R> *A) {
  const int nb = MU < 3 ? t * c.Lcu + sfwd<(MU < 3 ? MU : 0)>(q, c.L)
                        : ((t + 1) % c.L[3]) * c.Lcu + q.i;
  cx<R> B[9], U[9];
  load9(c.g, c.V, nb, B);
  load_link(c.U, c.V, MU, s, U);
  gtransform(A, U, B);
  store_link(c.U, c.V, MU, s, U);
}

template <typename R>
__global__ void __launch_bounds__(kCoulThreads) k_cslice_transform(CCtx<R> c,
                                                                   int all_t) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.V) return;
  const int t = s / c.Lcu;
  const SliceSite q = slice_site(s - t * c.Lcu, c.L);
  cx<R> A[9];
  load9(c.g, c.V, s, A);
  cslice_link<R, 0>(c, q, s, t, A);
  cslice_link<R, 1>(c, q, s, t, A);
  cslice_link<R, 2>(c, q, s, t, A);
  if (all_t || t < c.L[3] - 1) cslice_link<R, 3>(c, q, s, t, A);
}

// the temporal links of the last local slice, U_t <- g_last U_t g_next^dag,
// in the caller's AoS links (double[V][4][9][2]); g_last and g_next are the
// fields of that slice and of the following one (double[9][Lcu][2])
__global__ void __launch_bounds__(kCoulThreads)
    k_cfinish_aos(double2 *links, const double2 *g_last, const double2 *g_next,
                  int V, int Lcu) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Lcu) return;
  const int s = V - Lcu + i;
  cx<double> A[9], B[9], U[9];
#pragma unroll
  for (int e = 0; e < 9; e++) {
    const double2 a = g_last[(size_t)e * Lcu + i];
    const double2 b = g_next[(size_t)e * Lcu + i];
    A[e] = mk<double>(a.x, a.y);
    B[e] = mk<double>(b.x, b.y);
  }
  double2 *u = links + ((size_t)s * 4 + 3) * 9;
#pragma unroll
  for (int e = 0; e < 9; e++) U[e] = mk<double>(u[e].x, u[e].y);
  gtransform(A, U, B);
#pragma unroll
  for (int e = 0; e < 9; e++) u[e] = make_double2(U[e].x, U[e].y);
}

// g of local slice t, exported as double[9][Lcu][2]
__global__ void k_cexport_slice(const cx<double> *g, double2 *out, int V,
                                int Lcu, int t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Lcu) return;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    const cx<double> v = g[(size_t)e * V + (size_t)t * Lcu + i];
    out[(size_t)e * Lcu + i] = make_double2(v.x, v.y);
  }
}

template <typename R>
__global__ void k_cinit(CCtx<R> c) {
  const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (s >= (size_t)c.V) return;
  cx<R> G[9];
  set_identity(G);
  store9(c.g, c.V, (int)s, G);
}

}  // namespace gfix
