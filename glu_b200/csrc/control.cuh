// The control of the solvers on the device: the state of a Landau run and of
// the Coulomb slices, the fixed-order sums of the kernels' partials, and
// GLU's scalar control flow.
//
// The Landau kernels that sum over the lattice end in grid_sum: their blocks
// store their partials and take a ticket, the last of them adds the partials
// in a fixed order and its first thread applies the scalar step (theta and the
// stop test, beta, alpha*, the end of an iteration).  A kernel of its own for
// each of these four cost a launch and a cold one-block pass over the partials:
// 0.041 ms of a 1.34 ms iteration at 32^3 x 64, a third of one at 8^4.  A
// ticket costs its block a memory fence, so these grids are sized to the SMs
// and loop over the sites (with a block for every 128 sites the derivative
// took 0.200 instead of 0.162 ms at 32^3 x 64).  The FP64 probes have no
// registers for that loop: on lattices of more than one wave of their blocks
// k_scalar follows them.
#pragma once

#include "su3.cuh"

namespace gfix {

constexpr double kVal49 = 0.4444444444444444;  // lin_derivs.c:72
constexpr int kSiteThreads = 128;

enum ScalarOp : int {
  OP_THETA_TEST = 0,  // theta_test_lin = 2 sum / (NC V)
  OP_THETA_SD,        // theta of an SD start: reduction slots carry over
  OP_THETA_MAIN,      // theta at the top of a CG/SD iteration
  OP_PR,              // beta of the CG direction
  OP_PROBES,          // alpha* from the probes (or the fixed step)
  OP_DER,             // inold after the SD start
  OP_END_CG,          // end of a CG iteration
  OP_END_SD,          // end of an SD (FASD) iteration
  OP_NONE,            // no scalar step after this kernel
};

struct DevState {
  double tr;          // in-loop theta of the current iteration
  double tr_test;     // theta_test_lin
  double func;        // gauge functional of the current links
  double inold, insum, sumconj, beta, alpha;
  double ls_last[2];  // probe sums left in GLU's reduction slots
  double insum_last;  // insum left in GLU's reduction slot
  double gf_alpha, acc;
  long long max_iters;
  long long iter;     // loc_iters of the current run
  long long traj_len, traj_cap;
  double *traj_theta, *traj_func;
  int use_ls;         // this step uses the line search
  int stop;           // current iteration is the last one of the run
  int done;           // run finished: kernels return at once
  int upd;            // the link update of this iteration is due
  int parity;         // fb[parity] = in, fb[parity ^ 1] = in_old
  int sparity;        // sb[sparity] = sn (old), sb[sparity ^ 1] = new
  int sd_fixed;       // GLU_GFIX_SD: fixed step gf_alpha in SD steps
  double cg_tol;      // CG_TOL (GLU_definitions.h:451-455)
  double hp_below;    // FP32 storage: probes in FP64 arithmetic once tr < this
  // stall rule of a mixed-precision FP32 phase (stall_window 0: off): once
  // the best theta is below stall_floor, the run ends when theta has not
  // improved on it by 10% for stall_window iterations or exceeds blowup x it
  double best_tr, stall_floor, blowup;
  long long since_best, stall_window;
};

// which arithmetic variant of a kernel runs this step (FP32 storage: FP32
// arithmetic while theta >= hp_below, FP64 arithmetic below; a NaN theta
// takes the FP32 variant)
enum ArithSel : int { SEL_ALWAYS = 0, SEL_LOW = 1, SEL_HIGH = 2 };
__device__ __forceinline__ bool arith_skip(int sel, double tr, double below) {
  const bool high = tr < below;
  return (sel == SEL_LOW && high) || (sel == SEL_HIGH && !high);
}

// PREC_TOL (GLU_definitions.h:359-363): NC 1e-14 in double, NC 1e-6 in
// single precision builds
constexpr double kPrecTol = 3 * 1.0E-14;
constexpr double kPrecTolSingle = 3 * 1.0E-6;
constexpr int kCoulThreads = 128;

enum SliceMode : int { SL_RUN = 0, SL_DONE = 1 };

struct Slice {
  double tr, inold, insum, sumconj, beta, alpha;
  long long iter;     // steps of the current run (GLU's loc_iters)
  long long tot;      // GLU's tot_iters of steep_fix
  int sd;             // next step is an SD step
  int use_ls;
  int mode;           // SL_RUN / SL_DONE
  int control;        // random restarts so far
  int reunit;         // maintenance: reunitarise g_t and check it
  int randomize;      // maintenance: random restart of g_t
  int bad;            // set when the unitarity check fails
  int trans;          // GLU's trans_flag: survives a continuation run
  int traj_len;
  double best_tr;     // stall rule (mixed-precision FP32 phase)
  long long since_best;
};

struct CoulState {
  double gf_alpha, acc, cg_tol;
  long long max_iters;
  int facg;           // 1 FACG, 0 FASD
  int sd_fixed;       // GLU_GFIX_SD semantics
  int active;         // slices still running
  int nslices;
  unsigned long long seed;
  int traj_cap;       // per slice
  double *traj;       // [nslices][traj_cap]
  int *done_mask;     // [nslices], 1 once a slice has finished (FFT passes skip it)
  double prec_tol;    // PREC_TOL of the unitarity check
  double hp_below;    // FP32 storage: FP64 arithmetic for slices below this theta
  // stall rule of a mixed-precision FP32 phase (stall_window 0: off): a
  // slice whose best theta is below stall_floor ends its run after
  // stall_window iterations without a 10% improvement on it, or on a jump
  // above blowup x it; the FP64 phase then continues it
  long long stall_window;
  double stall_floor, blowup;
};

// ---------------------------------------------------------------------
// sums

// sum over the warp, in lane 0
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// the same over its first n lanes, where no others are
__device__ __forceinline__ double warp_sum(double v, int n) {
  const int lane = threadIdx.x & 31;
  const unsigned m = n >= 32 ? 0xffffffffu : (1u << n) - 1u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_down_sync(m, v, o);
    if (lane + o < n) v += t;
  }
  return v;
}

// deterministic block sum of NV values; thread 0 writes them to out[0..NV).
// RAGGED: the block may not be whole warps.
template <int NV, bool RAGGED = false>
__device__ __forceinline__ void block_sum_store(double (&v)[NV], double *out) {
  __shared__ double sh[NV][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  const int nl = RAGGED ? min(32, (int)blockDim.x - (warp << 5)) : 32;
#pragma unroll
  for (int k = 0; k < NV; k++) v[k] = RAGGED ? warp_sum(v[k], nl) : warp_sum(v[k]);
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) sh[k][warp] = v[k];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double x;
      if constexpr (RAGGED) {
        x = 0.0;
        for (int w = lane; w < nw; w += nl) x += sh[k][w];
        x = warp_sum(x, nl);
      } else {
        x = warp_sum(lane < nw ? sh[k][lane] : 0.0);
      }
      if (lane == 0) out[k] = x;
    }
  }
}

// True in every thread of the block that is the last of n to come here; the
// writes of all n blocks before it are then visible.  The ticket returns to
// zero.
__device__ __forceinline__ bool arrive_last(unsigned *tick, unsigned n) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(tick, 1u) == n - 1;
    if (last) *tick = 0;
  }
  __syncthreads();
  const bool l = last != 0;
  if (l) __threadfence();
  return l;
}

// blocks come in groups, so that the last block's pass over the partials
// does not grow with the lattice where a grid does (the xy passes)
constexpr unsigned kTickGroup = 1024;
__host__ __device__ constexpr unsigned tick_groups(unsigned nb) {
  return (nb + kTickGroup - 1) / kTickGroup;
}

// Totals of the pairs v over nb blocks, in fixed order: grid_sum is true in
// thread 0 of the last block, which then holds them in v.  part: nb pairs and
// after them one pair for each group.  A block may have work of its own
// between the two calls, whose stores the ticket's fence then does not wait
// for.
__device__ __forceinline__ int *ticket_flag() {
  __shared__ int last;
  return &last;
}
template <bool RAGGED = false>
__device__ __forceinline__ void grid_sum_begin(double (&v)[2], double *part, unsigned *tick,
                                               unsigned b, unsigned nb) {
  const unsigned g = b / kTickGroup, n = min(kTickGroup, nb - g * kTickGroup);
  block_sum_store<2, RAGGED>(v, part + 2 * (size_t)b);
  if (threadIdx.x == 0) {
    __threadfence();
    const bool l = atomicAdd(tick + 1 + g, 1u) == n - 1;
    if (l) tick[1 + g] = 0;
    *ticket_flag() = l;
  }
}
__device__ __forceinline__ void sum_pairs(double (&v)[2], const double *p, unsigned n) {
  v[0] = v[1] = 0.0;
  for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
    v[0] += __ldcg(p + 2 * (size_t)i);
    v[1] += __ldcg(p + 2 * (size_t)i + 1);
  }
}
template <bool RAGGED = false>
__device__ __forceinline__ bool grid_sum(double (&v)[2], double *part, unsigned *tick,
                                         unsigned b, unsigned nb) {
  const unsigned g = b / kTickGroup, ng = tick_groups(nb);
  const unsigned g0 = g * kTickGroup, n = min(kTickGroup, nb - g0);
  double *gp = part + 2 * (size_t)nb;
  __shared__ double tot[2];
  __syncthreads();
  if (!*ticket_flag()) return false;
  __threadfence();
  sum_pairs(v, part + 2 * (size_t)g0, n);
  block_sum_store<2, RAGGED>(v, ng == 1 ? tot : gp + 2 * (size_t)g);
  if (ng > 1) {
    if (!arrive_last(tick, ng)) return false;
    sum_pairs(v, gp, ng);
    block_sum_store<2, RAGGED>(v, tot);
  }
  v[0] = tot[0];  // (thread 0 wrote them)
  v[1] = tot[1];
  return threadIdx.x == 0;
}

// ---------------------------------------------------------------------
// GLU's control flow

__device__ __forceinline__ double approx_minimum(const double *al,
                                                 const double *f) {
  // src/Gfix/line_search.c:38-57
  const double A = f[0] / ((al[0] - al[1]) * (al[0] - al[2]));
  const double B = f[1] / ((al[1] - al[0]) * (al[1] - al[2]));
  const double C = f[2] / ((al[2] - al[0]) * (al[2] - al[1]));
  const double Sol = (al[0] * (B + C) + al[1] * (A + C) + al[2] * (A + B)) /
                     (2 * (A + B + C));
  if (Sol > al[2]) return al[2];
  if (isnan(Sol) || isinf(Sol) || Sol < al[0]) return 0.08;
  return Sol;
}

// the scalar step `op` of a Landau run on the totals a0, a1 over V sites
__device__ inline void apply_scalar(DevState *st, int op, double a0, double a1, double V) {
  switch (op) {
    case OP_THETA_TEST:
      st->tr_test = 2.0 * a0 / (3.0 * V);
      st->func = 1.0 - a1 / (12.0 * V);
      break;
    case OP_THETA_SD:
    case OP_THETA_MAIN: {
      st->tr = a0 / (3.0 * V);  // GFNORM_LANDAU
      st->func = 1.0 - a1 / (12.0 * V);
      st->alpha = st->gf_alpha;  // the step of an SD iteration without probes
      st->upd = 1;
      if (st->traj_theta && st->traj_len < st->traj_cap) {
        st->traj_theta[st->traj_len] = st->tr;
        st->traj_func[st->traj_len] = st->func;
        st->traj_len++;
      }
      if (op == OP_THETA_MAIN) {
        // the top of a loop iteration zeroes GLU's reduction slots
        st->ls_last[0] = st->ls_last[1] = 0.0;
        st->stop = !((st->tr > st->acc) && (st->iter + 1 < st->max_iters));
        if (st->stall_window > 0) {
          if (st->tr < 0.9 * st->best_tr) {
            st->best_tr = st->tr;
            st->since_best = 0;
          } else {
            st->since_best++;
          }
          if (st->best_tr < st->stall_floor &&
              (st->since_best >= st->stall_window || st->tr > st->blowup * st->best_tr))
            st->stop = 1;
        }
      }
      break;
    }
    case OP_PR: {
      st->insum = a0;
      st->sumconj = a1;
      const double b = st->sumconj / st->inold;
      double beta = (b < 0.0) ? 0.0 : b;  // PRfmax (src/Gfix/CG.c:37-41)
      if (st->tr < st->cg_tol) beta = st->insum / st->inold;
      st->beta = beta;
      st->inold = st->insum;
      st->insum_last = st->insum;
      st->use_ls = st->tr > st->cg_tol;
      break;
    }
    case OP_PROBES: {
      if (st->use_ls) {
        const double d1 = a0 + st->ls_last[0], d2 = a1 + st->ls_last[1];
        st->ls_last[0] = d1;
        st->ls_last[1] = d2;
        const double al[3] = {0.0, 0.15, 0.30};
        const double f[3] = {0.0, -d1, -d2};
        st->alpha = approx_minimum(al, f);
      } else {
        st->alpha = st->gf_alpha;
      }
      break;
    }
    case OP_DER:
      st->inold = st->insum_last + a0;
      st->parity ^= 1;  // in_old = in
      break;
    case OP_END_CG:
      st->iter++;
      st->parity ^= 1;
      st->sparity ^= 1;
      if (st->stop) st->done = 1;
      break;
    case OP_END_SD:
      st->iter++;
      if (st->stop) st->done = 1;
      break;
  }
}

enum CoulOp : int { C_SUMS = 0, C_PROBES = 1, C_END1 = 2, C_END2 = 3 };

// the scalar step `op` of slice t (GLU's steep_step_FACG / _FASD and
// steep_fix, src/Gfix/CFACG.c:285-529) on the totals a0, a1 over it
__device__ inline void apply_slice(CoulState *cs, Slice *sl, DevState *st, int t, int op,
                                   double a0, double a1, double Lcu) {
  Slice &S = sl[t];
  switch (op) {
    case C_SUMS: {
      S.insum = a0;
      S.sumconj = a1;
      S.tr = a0 / (3.0 * Lcu);  // GFNORM_COULOMB
      if (S.sd) {
        S.inold = a0;
        S.beta = 0.0;
        // FACG's SD start always searches (CFACG.c:318); FASD steps
        // search unless GLU_GFIX_SD (CFACG.c:270-280)
        S.use_ls = cs->facg ? 1 : !cs->sd_fixed;
      } else {
        const double b = S.sumconj / S.inold;
        double beta = (b < 0.0) ? 0.0 : b;
        if (S.tr < cs->cg_tol) beta = S.insum / S.inold;
        S.beta = beta;
        S.inold = S.insum;
        S.use_ls = S.tr > cs->cg_tol;
      }
      if (cs->traj && S.traj_len < cs->traj_cap)
        cs->traj[(size_t)t * cs->traj_cap + S.traj_len++] = S.tr;
      break;
    }
    case C_PROBES: {
      if (S.use_ls) {
        const double al[3] = {0.0, 0.17, 0.34};
        const double f[3] = {0.0, -a0, -a1};
        S.alpha = approx_minimum(al, f);
      } else {
        S.alpha = cs->gf_alpha;
      }
      break;
    }
    case C_END1: {
      S.reunit = 0;
      S.bad = 0;
      S.randomize = 0;
      if (cs->facg && S.sd) {
        S.sd = 0;  // the SD start is not counted
        break;
      }
      S.iter++;
      if (cs->stall_window > 0 && S.tr > cs->acc) {
        if (S.tr < 0.9 * S.best_tr) {
          S.best_tr = S.tr;
          S.since_best = 0;
        } else {
          S.since_best++;
        }
        if (S.best_tr < cs->stall_floor &&
            (S.since_best >= cs->stall_window || S.tr > cs->blowup * S.best_tr)) {
          S.sd = -1;  // ends the run, no restart: the FP64 phase goes on
          break;
        }
      }
      if ((S.tr > cs->acc) && (S.iter < cs->max_iters)) break;
      S.reunit = S.tr < cs->acc;  // run ended: adequate_solution first
      S.sd = -1;                  // marks "ended" for C_END2
      break;
    }
    case C_END2: {
      if (S.sd != -1) break;
      const long long loc = S.iter;
      const bool fin = isfinite(S.tr);
      if (atomicOr(&S.bad, 0)) S.trans = 1;  // (set by this kernel's blocks)
      S.sd = 1;
      S.iter = 0;
      if (loc >= cs->max_iters) {
        if (S.tr < 1E4 * cs->acc && fin) {  // continuation run
          S.tot += loc;
          break;
        }
        if (S.tr > cs->acc || !fin) S.trans = 1;
      }
      if (S.control < 8 && S.trans) {  // random restart
        S.randomize = 1;
        S.trans = 0;
        S.tot += loc;
        S.control++;
        break;
      }
      S.tot += loc;
      S.iter = loc;
      S.mode = SL_DONE;
      cs->done_mask[t] = 1;
      // the slice that ends last stops the whole sequence
      if (atomicSub(&cs->active, 1) == 1) st->done = 1;
      break;
    }
  }
}

}  // namespace gfix
