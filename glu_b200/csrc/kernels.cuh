// Device kernels of the Fourier-accelerated Landau gauge fixing on B200.
//
// One iteration of FACG (src/Gfix/FACG.c:270-334) is the launch sequence
//   k_deriv          Delta(x) packed in 4 fields, then theta, functional and
//                    the stop decision
//   k_fft_xy  fwd    x,y passes of the 4D FFT, one xy-plane per block
//   k_fft_zt         z,t passes, * psq, inverse t,z passes (one tile/block)
//   k_fft_xy  bwd    inverse x,y passes fused with the PR sums, then beta
//                    (PR+ / FR switch at CG_TOL)
//   k_dir_probe      sn <- in + beta sn, line-search probes of GLU's
//                    line_search_Landau (src/Gfix/line_search.c:274-341), then
//                    alpha* by the parabola of approx_minimum; iteration
//                    count, buffer parities, done flag
//   k_update         U_mu(x) <- g(x) U_mu(x) g(x+mu)^dag, g = reunit(1+a A)
// The scalar steps are taken by the last block of each kernel (control.cuh),
// those after the FP64 probes of large lattices by k_scalar.
// Every kernel first checks the device-side done flag, so a captured graph
// of the iteration can be replayed past convergence as a no-op.
//
// HBM layout (SoA, site index s = x + Lx (y + Ly (z + Lz t))):
//   U   cx<R>[4 mu][6 elements][V]        links: their first two columns
//                                          (load_link rebuilds the third)
//   fb  cx<F>[2][4 fields][V]             in / in_old (parity selects)
//   sb  cx<F>[2][4 fields][V]             sn ping-pong (sparity selects)
//   G   cx<R>[9][V]                        accumulated gauge transform
//                                          (mixed precision only)
// R is the type of the links (and of the link arithmetic), F that of the
// su(3) fields and of the FFT: F = R except in the FP64 phase of a
// mixed-precision solve, which keeps FP64 links, theta and updates but
// carries its search directions and their Fourier acceleration in FP32.
#pragma once

#include "control.cuh"
#include "fft.cuh"

namespace gfix {

// set or clear the done flag (used to run every kernel once as a no-op)
static __global__ void k_set_done(DevState *st, int v) { st->done = v; }

// start of a solver run (GLU's steep_Landau_FACG / _FASD entry)
static __global__ void k_begin_run(DevState *st) {
  st->iter = 0;
  st->done = 0;
  st->stop = 0;
  st->use_ls = !st->sd_fixed;
}

template <typename R, typename F = R>
struct Ctx {
  cx<R> *U;
  cx<F> *fb[2];
  cx<F> *sb[2];
  cx<R> *G;
  DevState *st;
  double *part;       // [nblocks][2] per-block partial sums, group totals
  unsigned *tick;     // tickets of grid_sum, zero between kernels
  const cx<F> *tw;    // twiddle pool
  const double *cs;   // cos tables, cs[mu * cs_ld + n] = cos(n 2pi/L_mu)
  int cs_ld;
  int L[4];
  int V;
  int ndim;           // FFT rank: 4 Landau, 3 Coulomb
  int zt_b;           // x columns per zt tile
  int xy_pitch;       // padded row pitch of the xy tile
  double maxp;        // MAX_LANDAU = 4 ND / V or MAX_COULOMB = 4 (ND-1)/Lcu
  FftAxis ax[4];
  const int *skip;    // ndim 3: per-slice flags, set slices are not transformed
  CoulState *cst;     // ndim 3: control of the slices, and a ticket for each
  Slice *csl;
  unsigned *ctick;
};

// ---------------------------------------------------------------------
// helpers

// buffer of a ping-pong pair by parity, as a select (a runtime index into
// the by-value kernel parameter would copy it to local memory)
template <typename T>
__device__ __forceinline__ T *pick(T *const (&b)[2], int p) {
  return p ? b[1] : b[0];
}

__device__ __forceinline__ void coords(int s, const int *L, int *x) {
  x[0] = s % L[0];
  s /= L[0];
  x[1] = s % L[1];
  s /= L[1];
  x[2] = s % L[2];
  x[3] = s / L[2];
}

__device__ __forceinline__ int fwd_site(int s, int mu, const int *x,
                                        const int *L, const int *stride) {
  return x[mu] == L[mu] - 1 ? s - (L[mu] - 1) * stride[mu] : s + stride[mu];
}
// fwd_site for a run-time direction, by selects in registers
__device__ __forceinline__ int fwd_rt(int s, int mu, const int *x, const int *L,
                                      const int *stride) {
  const int xm = mu == 0 ? x[0] : mu == 1 ? x[1] : mu == 2 ? x[2] : x[3];
  const int lm = mu == 0 ? L[0] : mu == 1 ? L[1] : mu == 2 ? L[2] : L[3];
  const int sm = mu == 0 ? stride[0] : mu == 1 ? stride[1] : mu == 2 ? stride[2] : stride[3];
  return xm == lm - 1 ? s - (lm - 1) * sm : s + sm;
}
__device__ __forceinline__ int bck_site(int s, int mu, const int *x,
                                        const int *L, const int *stride) {
  return x[mu] == 0 ? s + (L[mu] - 1) * stride[mu] : s - stride[mu];
}

template <typename CT>
__device__ __forceinline__ void strides(const CT &c, int *st) {
  st[0] = 1;
  st[1] = c.L[0];
  st[2] = c.L[0] * c.L[1];
  st[3] = c.L[0] * c.L[1] * c.L[2];
}

// Links in HBM keep their first two columns only: the complex entries
// 0, 1, 3, 4, 6, 7 of the row-major matrix, stored U[mu][k][V], k = 0..5
// (96 of a link's 144 bytes in FP64).  The third column is rebuilt on every
// load as the conjugate cross product of the first two -- the expression
// with which GLU's update (gtransform, src/Gfix/gtrans.c:107-121) and this
// library's own (su3.cuh) complete every link they write -- so a link that
// has been updated once reads back bit for bit as it was computed, and an
// SU(3) input differs from its stored third column by rounding only.
constexpr int kLinkCx = 6;

template <typename R>
__device__ __forceinline__ void load_link(const cx<R> *U, int V, int mu, int s,
                                          cx<R> *u) {
  const cx<R> *p = U + (size_t)mu * kLinkCx * V + s;
  u[0] = p[0];
  u[1] = p[(size_t)V];
  u[3] = p[2 * (size_t)V];
  u[4] = p[3 * (size_t)V];
  u[6] = p[4 * (size_t)V];
  u[7] = p[5 * (size_t)V];
  complete_col2(u);
}

// the stored first two columns alone
template <typename R>
__device__ __forceinline__ void load_cols(const cx<R> *U, int V, int mu, int s,
                                          cx<R> *u0, cx<R> *u1) {
  const cx<R> *p = U + (size_t)mu * kLinkCx * V + s;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    u0[r] = p[2 * r * (size_t)V];
    u1[r] = p[(2 * r + 1) * (size_t)V];
  }
}

template <typename R>
__device__ __forceinline__ void store_link(cx<R> *U, int V, int mu, int s,
                                           const cx<R> *u) {
  cx<R> *p = U + (size_t)mu * kLinkCx * V + s;
  p[0] = u[0];
  p[(size_t)V] = u[1];
  p[2 * (size_t)V] = u[3];
  p[3 * (size_t)V] = u[4];
  p[4 * (size_t)V] = u[6];
  p[5 * (size_t)V] = u[7];
}

// ---------------------------------------------------------------------
// K1: the gauge derivative, fused with the theta and functional sums
// (src/Gfix/lin_derivs.c:74-193 packed as src/Gfix/FACG.c:54-60)

template <typename R, typename F = R>
__global__ void __launch_bounds__(kSiteThreads, sizeof(R) == 8 ? 5 : 7)
    k_deriv(Ctx<R, F> c, int op) {
  if (c.st->done) return;
  double v[2] = {0.0, 0.0};
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < c.V; s += gridDim.x * blockDim.x) {
    int x[4], sd[4];
    coords(s, c.L, x);
    strides(c, sd);
    R R0 = 0, R1 = 0, I1 = 0, R2 = 0, I2 = 0, R3 = 0, R4 = 0, I4 = 0;
    double re = 0.0;
#pragma unroll
    for (int mu = 0; mu < 4; mu++) {
      cx<R> q[9], b[9];
      load_link(c.U, c.V, mu, s, q);
      load_link(c.U, c.V, mu, bck_site(s, mu, x, c.L, sd), b);
      const cx<R> q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4],
                  q5 = q[5], q6 = q[6], q7 = q[7], q8 = q[8];
      const cx<R> b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3], b4 = b[4],
                  b5 = b[5], b6 = b[6], b7 = b[7], b8 = b[8];
      R0 += R(2) * b0.y - b4.y - b8.y;
      R0 += R(-2) * q0.y + q4.y + q8.y;
      R1 += b1.x - b3.x - q1.x + q3.x;
      I1 += b1.y + b3.y - q1.y - q3.y;
      R2 += b2.x - b6.x - q2.x + q6.x;
      I2 += b2.y + b6.y - q2.y - q6.y;
      R3 += R(2) * b4.y - b0.y - b8.y;
      R3 += R(-2) * q4.y + q0.y + q8.y;
      R4 += b5.x - b7.x - q5.x + q7.x;
      I4 += b5.y + b7.y - q5.y - q7.y;
      re += (double)q0.x + (double)q4.x + (double)q8.x;
    }
    cx<F> *f = c.fb[c.st->parity];
    const size_t V = c.V;
    f[s] = mk<F>((F)(-(R3 / R(3))), (F)(R0 / R(3)));
    f[V + s] = mk<F>((F)(R(0.5) * R1), (F)(R(0.5) * I1));
    f[2 * V + s] = mk<F>((F)(R(0.5) * R2), (F)(R(0.5) * I2));
    f[3 * V + s] = mk<F>((F)(R(0.5) * R4), (F)(R(0.5) * I4));
    const double d0 = R0, d1 = R1, e1 = I1, d2 = R2, e2 = I2, d3 = R3,
                 d4 = R4, e4 = I4;
    v[0] += kVal49 * (d0 * d0 + d3 * (d3 + d0)) +
           (d1 * d1 + e1 * e1 + d2 * d2 + e2 * e2 + d4 * d4 + e4 * e4);
    v[1] += re;
  }
  grid_sum_begin(v, c.part, c.tick, blockIdx.x, gridDim.x);
  if (grid_sum(v, c.part, c.tick, blockIdx.x, gridDim.x))
    apply_scalar(c.st, op, v[0], v[1], (double)c.V);
}

// ---------------------------------------------------------------------
// the 4D (or batched 3D) FFT with psq folded into the middle pass

#include "fft_pass.cuh"
#include "fft_ct.cuh"

// ---------------------------------------------------------------------
// K4: conjugate direction update fused with the line-search probes.
// DIR: sn_new = in + beta sn_old (src/Gfix/FACG.c:315-323), else the
// direction is `in` itself (an SD step).  Probes: per site the three
// values of src/Gfix/line_search.c:296-313 at alpha = 0, 0.15, 0.30;
// accumulated as differences to the alpha = 0 value, which leaves the
// parabola of approx_minimum unchanged and avoids cancelling large sums.

// the direction at site s as stored (type F): computed in R, rounded to F;
// f receives it back in R, so the probes use the direction the update reads
template <typename R, bool DIR, typename F>
__device__ __forceinline__ void dir_at(const Ctx<R, F> &c, const cx<F> *in,
                                       const cx<F> *so, R beta, int s,
                                       cx<R> *f, cx<F> *fs = nullptr) {
  const size_t V = c.V;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const cx<F> a = in[k * V + s];
    cx<F> r;
    if (DIR) {
      const cx<F> b = so[k * V + s];
      r = mk<F>((F)fma(beta, (R)b.x, (R)a.x), (F)fma(beta, (R)b.y, (R)a.y));
    } else {
      r = a;
    }
    if (fs) fs[k] = r;
    f[k] = mk<R>((R)r.x, (R)r.y);
  }
}

// C is the arithmetic precision of the probes: the FP32 phase of the mixed
// solver evaluates them in FP64 from its FP32 links and directions once
// theta < hp_below (1e-5), because per-site probe differences fall below
// FP32 rounding once theta < ~1e-6; above it FP32 arithmetic serves.  Both
// variants are launched, `sel` lets the one that fits the step run.
//
// Bound by FP64 arithmetic.  A direction's link and neighbour are loaded once
// for both probes, with the site's own matrices waiting in shared memory, and
// the traces go by probe_trace: 1,800 operations a site where forming every
// g(x + mu) and the third columns took 2,400.  At 32^3 x 64, per launch:
// 0.462 -> 0.361 ms in FP64, 0.478 -> 0.390 ms with FP32 fields, 0.261 ->
// 0.23 ms in FP32.  Blocks per SM: four (128 registers) in FP64, three take
// 0.393 ms; six in FP32, four 0.237 ms.  Both probes unrolled together spill
// (0.685 ms).
template <typename R, bool DIR, typename C, typename F, bool FUSED>
__global__ void __launch_bounds__(kSiteThreads, sizeof(C) == 4 ? 6 : 4) k_dir_probe(Ctx<R, F> c, int sel, int end) {
  if (c.st->done || arith_skip(sel, c.st->tr, c.st->hp_below)) return;
  __shared__ cx<C> sA[2][9][kSiteThreads];  // g(x) at both probes
  const int par = c.st->parity, spar = c.st->sparity;
  const cx<F> *in = pick(c.fb, par);
  const cx<F> *so = pick(c.sb, spar);
  cx<F> *sn = pick(c.sb, spar ^ 1);
  const R beta = (R)c.st->beta;
  const bool probes = c.st->use_ls != 0;
  double v[2] = {0.0, 0.0};
  const int s0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int s = s0; s < c.V; s += gridDim.x * blockDim.x) {
    cx<R> f[4];
    cx<F> fs[4];
    dir_at<R, DIR>(c, in, so, beta, s, f, fs);
    if (DIR) {
#pragma unroll
      for (int k = 0; k < 4; k++) sn[(size_t)k * c.V + s] = fs[k];
    }
    if (probes) {
      int x[4], sd[4];
      coords(s, c.L, x);
      strides(c, sd);
      auto up = [](cx<R> a) { return mk<C>((C)a.x, (C)a.y); };
#pragma unroll 1
      for (int k = 0; k < 2; k++) {
        cx<C> A[9];
        set_gauge(A, up(f[0]), up(f[1]), up(f[2]), up(f[3]), k == 0 ? C(0.15) : C(0.30));
#pragma unroll
        for (int e = 0; e < 9; e++) sA[k][e][threadIdx.x] = A[e];
      }
      C d[2] = {0, 0};
#pragma unroll 1
      for (int mu = 0; mu < 4; mu++) {
        const int y = fwd_rt(s, mu, x, c.L, sd);
        cx<R> fy[4], u0[3], u1[3];
        dir_at<R, DIR>(c, in, so, beta, y, fy);
        load_cols(c.U, c.V, mu, s, u0, u1);
        cx<C> w0[3], w1[3];
#pragma unroll
        for (int r = 0; r < 3; r++) w0[r] = up(u0[r]), w1[r] = up(u1[r]);
        const C t0 = re_tr_cols(w0, w1);
        const ProbeDir<C> p = probe_dir(up(fy[0]), up(fy[1]), up(fy[2]), up(fy[3]));
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
          cx<C> A[9];
#pragma unroll
          for (int e = 0; e < 9; e++) A[e] = sA[k][e][threadIdx.x];
          d[k] += probe_trace(A, w0, w1, p, k == 0 ? C(0.15) : C(0.30)) - t0;
        }
      }
      v[0] += d[0];
      v[1] += d[1];
    }
    if (!FUSED) break;
  }
  if constexpr (!FUSED) {
    if (probes) block_sum_store<2>(v, c.part + 2 * blockIdx.x);
    return;
  }
  grid_sum_begin(v, c.part, c.tick, blockIdx.x, gridDim.x);
  if (grid_sum(v, c.part, c.tick, blockIdx.x, gridDim.x)) {
    apply_scalar(c.st, OP_PROBES, v[0], v[1], (double)c.V);
    apply_scalar(c.st, end, 0.0, 0.0, (double)c.V);
  }
}

// the probes' scalar step by a kernel of its own, where their grid has a block
// for every 128 sites of a large lattice and a ticket for each would cost
// more; sel: of the probes' variant.  op: OP_PROBES with `end`, or OP_NONE with
// `end` alone
constexpr int kScalarThreads = 1024;
static __global__ void __launch_bounds__(kScalarThreads)
    k_scalar(DevState *st, const double *part, int nb, int sel, int op, int end, double V) {
  if (st->done || arith_skip(sel, st->tr, st->hp_below)) return;
  double v[2] = {0.0, 0.0};
  if (op != OP_NONE) {
    // eight independent loads in flight per thread and round, then added in a
    // fixed order
    constexpr int kU = 8;
    const double2 *p = reinterpret_cast<const double2 *>(part);
    for (int i0 = threadIdx.x; i0 < nb; i0 += kU * kScalarThreads) {
      double2 x[kU];
#pragma unroll
      for (int k = 0; k < kU; k++) {
        const int i = i0 + k * kScalarThreads;
        x[k] = i < nb ? p[i] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int k = 0; k < kU; k++) {
        v[0] += x[k].x;
        v[1] += x[k].y;
      }
    }
    __shared__ double tot[2];
    block_sum_store<2>(v, tot);
    v[0] = tot[0];
    v[1] = tot[1];
  }
  if (threadIdx.x != 0) return;
  apply_scalar(st, op, v[0], v[1], V);
  apply_scalar(st, end, 0.0, 0.0, V);
}


// ---------------------------------------------------------------------
// K5: the link update of egauge_Landau (src/Gfix/line_search.c:60-97):
// g(x) = reunit(1 + alpha A(x)), U_mu(x) <- g(x) U_mu(x) g(x+mu)^dag.
// SN selects the direction: the new conjugate direction or `in` (the end of
// the iteration, which flips sn's buffers, has been applied with the probes').
// With G (mixed precision) the transform is accumulated, G(x) <- g(x) G(x).
//
// A link's third column is completed from its first two (as GLU does), so a
// departure from SU(3) passes on multiplied: by up to 4/3 for gauge rotations
// of order one, less on a plateau.  Left alone it reaches 5e-8 after 900
// iterations at 32^3 x 64 and takes a fix of 48^3 x 96 off its gauge orbit
// (plaquette 6e-8 off); so FP64 links are reunitarised every kReunitEvery
// iterations, in which a departure grows tenfold at most.  (FP32 links are not:
// the phase they serve ends on the FP64 input's orbit in any case, and took
// more iterations with it.)
//
// Bound by the bytes of links and fields.  In FP64 the registers allow three
// blocks per SM, whose loads alone don't cover the latency between two
// directions: each thread fetches the next direction's link and neighbour to
// shared memory while it works on this one.  32^3 x 64: 0.326 -> 0.287 ms
// (0.93 of the copy bandwidth; FP32 fields 0.321 -> 0.285), 48^3 x 96 1.676 ->
// 1.418 (0.95), 24^3 x 48 0.110 -> 0.095.  FP32 links are at 0.94 to 0.97 as
// they are.

constexpr int kReunitEvery = 8;

template <typename R, bool SN, typename F = R>
__global__ void __launch_bounds__(kSiteThreads) k_update(Ctx<R, F> c) {
  if (!c.st->upd) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.V) return;
  const cx<F> *d = SN ? c.sb[c.st->sparity] : c.fb[c.st->parity];
  const R alpha = (R)c.st->alpha;
  const size_t V = c.V;
  int x[4], sd[4];
  coords(s, c.L, x);
  strides(c, sd);
  auto up = [](cx<F> a) { return mk<R>((R)a.x, (R)a.y); };
  cx<R> A[9], Bm[9], U[9];
  if constexpr (sizeof(R) == 8) {
    // the next direction's link and neighbour on their way while this one is
    // worked (each thread its own)
    __shared__ cx<R> sU[kLinkCx][kSiteThreads];
    __shared__ cx<F> sF[4][kSiteThreads];
    const int tid = threadIdx.x;
    const bool reunit = c.st->iter % kReunitEvery == kReunitEvery - 1;
    auto fetch = [&](int mu) {
      const int y = fwd_site(s, mu, x, c.L, sd);
#pragma unroll
      for (int e = 0; e < kLinkCx; e++)
        cp_async(&sU[e][tid], c.U + ((size_t)mu * kLinkCx + e) * V + s);
#pragma unroll
      for (int k = 0; k < 4; k++) cp_async(&sF[k][tid], d + k * V + y);
    };
    fetch(0);
    set_gauge(A, up(d[s]), up(d[V + s]), up(d[2 * V + s]), up(d[3 * V + s]), alpha);
#pragma unroll 1
    for (int mu = 0; mu < 4; mu++) {
      cp_async_wait();
      cx<F> f[4];
#pragma unroll
      for (int k = 0; k < 4; k++) f[k] = sF[k][tid];
#pragma unroll
      for (int r = 0; r < 3; r++) U[3 * r] = sU[2 * r][tid], U[3 * r + 1] = sU[2 * r + 1][tid];
      __syncwarp(__activemask());  // (read before they are overwritten)
      if (mu < 3) fetch(mu + 1);
      complete_col2(U);
      set_gauge(Bm, up(f[0]), up(f[1]), up(f[2]), up(f[3]), alpha);
      gtransform(A, U, Bm);
      if (reunit) gram_reunit(U);
      store_link(c.U, c.V, mu, s, U);
    }
  } else {
    set_gauge(A, up(d[s]), up(d[V + s]), up(d[2 * V + s]), up(d[3 * V + s]), alpha);
#pragma unroll 1
    for (int mu = 0; mu < 4; mu++) {
      const int y = fwd_site(s, mu, x, c.L, sd);
      set_gauge(Bm, up(d[y]), up(d[V + y]), up(d[2 * V + y]), up(d[3 * V + y]), alpha);
      load_link(c.U, c.V, mu, s, U);
      gtransform(A, U, Bm);
      store_link(c.U, c.V, mu, s, U);
    }
  }
  if (c.G) {
    cx<R> g[9], r[9];
#pragma unroll
    for (int e = 0; e < 9; e++) g[e] = c.G[(size_t)e * V + s];
    multab(r, A, g);
#pragma unroll
    for (int e = 0; e < 9; e++) c.G[(size_t)e * V + s] = r[e];
  }
}

// sn = in_old = in after an SD start, with sum_DER3 (src/Gfix/FACG.c:148-178)
template <typename R>
__global__ void __launch_bounds__(256) k_copy_der(Ctx<R> c) {
  if (c.st->done) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const cx<R> *in = c.fb[c.st->parity];
  cx<R> *sn = c.sb[c.st->sparity];
  double v[2] = {0.0, 0.0};
  if (s < c.V) {
    double l = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const cx<R> a = in[(size_t)k * c.V + s];
      sn[(size_t)k * c.V + s] = a;
      const double ar = a.x, ai = a.y;
      l += (k == 0) ? (ar * ar + ai * ai + ar * ai) : (ar * ar + ai * ai);
    }
    v[0] = 2.0 * l;
  }
  grid_sum_begin(v, c.part, c.tick, blockIdx.x, gridDim.x);
  if (grid_sum(v, c.part, c.tick, blockIdx.x, gridDim.x))
    apply_scalar(c.st, OP_DER, v[0], v[1], (double)c.V);
}

// ---------------------------------------------------------------------
// layout conversion: host AoS double[V][4][9][2] <-> device SoA cx<R>

// One block moves kTrSites consecutive sites through shared memory so that
// both the AoS side (36 contiguous complex numbers per site) and the SoA side
// (kTrSites contiguous numbers per element row) are accessed coalesced.
constexpr int kTrSites = 64;

// matrix entry of stored element k of a link (its first two columns)
__device__ __forceinline__ int stored_entry(int k) { return (k >> 1) * 3 + (k & 1); }

template <typename R>
__global__ void __launch_bounds__(256) k_aos_to_soa(const double *__restrict__ aos,
                                                    cx<R> *U, int V) {
  __shared__ double2 t[kTrSites * 36 + 1];
  const size_t s0 = (size_t)blockIdx.x * kTrSites;
  const int ns = (int)min((size_t)kTrSites, (size_t)V - s0);
  const double2 *src = reinterpret_cast<const double2 *>(aos) + s0 * 36;
  for (int i = threadIdx.x; i < ns * 36; i += blockDim.x) t[i] = src[i];
  __syncthreads();
  // row r of the SoA links: direction r / 6, stored element r % 6
  for (int i = threadIdx.x; i < 4 * kLinkCx * kTrSites; i += blockDim.x) {
    const int r = i / kTrSites, sl = i % kTrSites;
    if (sl < ns) {
      const double2 v = t[sl * 36 + (r / kLinkCx) * 9 + stored_entry(r % kLinkCx)];
      U[(size_t)r * V + s0 + sl] = mk<R>((R)v.x, (R)v.y);
    }
  }
}

// one thread per (site, direction) of the block's kTrSites sites: the link
// completed in R (third column rebuilt as in load_link), then staged in
// shared memory for coalesced AoS stores
template <typename R>
__global__ void __launch_bounds__(256) k_soa_to_aos(const cx<R> *U,
                                                    double *__restrict__ aos,
                                                    int V) {
  __shared__ double2 t[kTrSites * 36 + 1];
  const size_t s0 = (size_t)blockIdx.x * kTrSites;
  const int ns = (int)min((size_t)kTrSites, (size_t)V - s0);
  for (int i = threadIdx.x; i < 4 * kTrSites; i += blockDim.x) {
    const int mu = i / kTrSites, sl = i % kTrSites;
    if (sl < ns) {
      cx<R> u[9];
      load_link(U, V, mu, (int)(s0 + sl), u);
#pragma unroll
      for (int e = 0; e < 9; e++)
        t[sl * 36 + mu * 9 + e] = make_double2((double)u[e].x, (double)u[e].y);
    }
  }
  __syncthreads();
  double2 *dst = reinterpret_cast<double2 *>(aos) + s0 * 36;
  for (int i = threadIdx.x; i < ns * 36; i += blockDim.x) dst[i] = t[i];
}

}  // namespace gfix
