// FFT passes whose threads hold whole pencils in registers.
//
// The passes of fft_ct.cuh give each thread one radix-8 butterfly and go
// through shared memory, with two barriers, between every two stages: a
// 32 x 64 (z,t) tile makes six such trips, and their address arithmetic,
// twiddle loads and barriers take longer than its transforms or its bytes
// (FP64: one block of 1024 threads fills an SM, so that nothing runs while
// it waits).  Here a thread transforms a pencil of up to 64 (FP32) or 32
// (FP64) elements in its registers, every index and twiddle a compile-time
// constant, and shared memory is crossed only to turn from one axis to the
// other: twice in a (z,t) pass, twice in an xy pass, never in the z pass of
// Coulomb slices, whose pencils neighbouring threads read in full lines.
// A t axis too long for one thread is split over two, t = 2n + h, which
// exchange half of their elements by shuffles (radix 2) on either side of
// the psq scale; the longest z and t axes over two and four.
//
// Per launch at 32^3 x 64: xy 0.070 -> 0.049 ms in FP64 (0.84 of the copy
// bandwidth), 0.039 -> 0.026 ms in FP32; inverse with sums 0.105 -> 0.087 and
// 0.069 -> 0.053 ms; (z, t) 0.167 -> 0.157 and 0.094 -> 0.066 ms.  FP32 at 48^3
// x 96: 0.260 -> 0.133, 0.437 -> 0.246 and 0.780 -> 0.492 ms.  FP64 at 20^3 x
// 40, where only the generic passes served: 0.070 + 0.120 + 0.082 -> 0.014 +
// 0.022 + 0.024 ms.  The register budget ends it: pencils of 64 in FP32 and 32
// in FP64 (planes of up to 64 by two lanes a
// pencil), Coulomb z pencils (no shared memory to share the work) of 48 and
// 24 (0.072 against 0.069 ms with 32 in FP64); beyond, fft_ct.cuh.
//
// Included by the FFT translation units (fft_xy_f32.cu .. fft_zt_f64.cu) only.
#pragma once

#include "kernels.cuh"

namespace gfix {

// --- compile-time cosines and sines of 2 pi p / q -------------------------
// (Taylor series on the first octant: below one unit in the last place)
__host__ __device__ constexpr double taylor(double x, bool cosine) {
  const double x2 = x * x;
  double term = cosine ? 1.0 : x, sum = 0.0;
  double t[14] = {};
  for (int k = 0; k < 14; k++) {
    t[k] = term;
    const int m = 2 * k + (cosine ? 1 : 2);
    term *= -x2 / (m * (m + 1.0));
  }
  for (int k = 13; k >= 0; k--) sum += t[k];  // smallest first
  return sum;
}
__host__ __device__ constexpr double sin_2pi(int p, int q);
__host__ __device__ constexpr double cos_2pi(int p, int q) {
  p = (p % q + q) % q;
  if (2 * p > q) p = q - p;
  if (4 * p > q) return -cos_2pi(q - 2 * p, 2 * q);
  if (8 * p > q) return sin_2pi(q - 4 * p, 4 * q);
  return taylor(6.283185307179586476925286766559 * p / q, true);
}
__host__ __device__ constexpr double sin_2pi(int p, int q) {
  p = (p % q + q) % q;
  if (2 * p > q) return -sin_2pi(q - p, q);
  if (4 * p > q) return sin_2pi(q - 2 * p, 2 * q);
  if (8 * p > q) return cos_2pi(q - 4 * p, 4 * q);
  return taylor(6.283185307179586476925286766559 * p / q, false);
}

// a constant of a type of its own, and f(Ic<0>) .. f(Ic<N - 1>)
template <int I>
struct Ic {
  __host__ __device__ constexpr operator int() const { return I; }
};
template <int N, int I = 0, class F>
__device__ __forceinline__ void static_for(F &&f) {
  if constexpr (I < N) {
    f(Ic<I>{});
    static_for<N, I + 1>(f);
  }
}

// v e^{-+ 2 pi i K / N} (B: +)
template <typename R, int K, int N, bool B>
__device__ __forceinline__ cx<R> rot(cx<R> v) {
  constexpr int k = K % N;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (2 * k == N) {
    return mk<R>(-v.x, -v.y);
  } else if constexpr (4 * k == N) {
    return B ? mk<R>(-v.y, v.x) : mk<R>(v.y, -v.x);
  } else if constexpr (4 * k == 3 * N) {
    return B ? mk<R>(v.y, -v.x) : mk<R>(-v.y, v.x);
  } else {
    constexpr R c = (R)cos_2pi(k, N), s = (R)(B ? sin_2pi(k, N) : -sin_2pi(k, N));
    if constexpr (8 * k == N || 8 * k == 3 * N || 8 * k == 5 * N || 8 * k == 7 * N) {
      // |c| = |s|
      constexpr R h = (R)cos_2pi(1, 8);
      constexpr bool cp = c > R(0), sp = s > R(0);
      const R a = (cp ? v.x : -v.x) - (sp ? v.y : -v.y);
      const R b = (sp ? v.x : -v.x) + (cp ? v.y : -v.y);
      return mk<R>(h * a, h * b);
    }
    return mk<R>(fma(v.x, c, -(v.y * s)), fma(v.x, s, v.y * c));
  }
}

// in-register DFT of v, natural order in and out, unnormalised
template <typename R, int N, bool B>
struct RegFft {
  __host__ __device__ static constexpr int split() {
    if (N % 8 == 0 && N > 16) return 8;
    if (N % 4 == 0) return 4;
    for (int r = 2; r < N; r++)
      if (N % r == 0) return r;
    return N;
  }
  __device__ __forceinline__ static void run(cx<R> (&v)[N]) {
    if constexpr (N == 1) {
    } else if constexpr (N == 2) {
      const cx<R> a = v[0];
      v[0] = cadd(a, v[1]);
      v[1] = csub(a, v[1]);
    } else if constexpr (N == 4) {
      const cx<R> a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
      const cx<R> c = cadd(v[1], v[3]), d = rot<R, 1, 4, B>(csub(v[1], v[3]));
      v[0] = cadd(a, c);
      v[1] = cadd(b, d);
      v[2] = csub(a, c);
      v[3] = csub(b, d);
    } else if constexpr (split() == N) {
      // odd prime: cosine sums of v_j + v_{N-j}, sine sums of v_j - v_{N-j}
      constexpr int H = N / 2;
      cx<R> s[H], d[H], out[N];
      static_for<H>([&](auto J) {
        constexpr int j = J;
        s[j] = cadd(v[j + 1], v[N - 1 - j]);
        d[j] = csub(v[j + 1], v[N - 1 - j]);
      });
      out[0] = v[0];
      static_for<H>([&](auto J) { out[0] = cadd(out[0], s[J]); });
      static_for<H>([&](auto K) {
        constexpr int k = K + 1;
        cx<R> c = v[0], t = mk<R>(R(0), R(0));
        static_for<H>([&](auto J) {
          constexpr int j = J;
          constexpr R wc = (R)cos_2pi((j + 1) * k, N), ws = (R)sin_2pi((j + 1) * k, N);
          c = mk<R>(fma(s[j].x, wc, c.x), fma(s[j].y, wc, c.y));
          t = mk<R>(fma(d[j].x, ws, t.x), fma(d[j].y, ws, t.y));
        });
        // e^{-i}: c - i t, e^{+i}: c + i t
        out[k] = B ? mk<R>(c.x - t.y, c.y + t.x) : mk<R>(c.x + t.y, c.y - t.x);
        out[N - k] = B ? mk<R>(c.x + t.y, c.y - t.x) : mk<R>(c.x - t.y, c.y + t.x);
      });
      static_for<N>([&](auto J) { v[J] = out[J]; });
    } else {
      constexpr int N1 = split(), N2 = N / N1;
      static_for<N2>([&](auto I) {
        constexpr int n2 = I;
        cx<R> a[N1];
        static_for<N1>([&](auto J) { a[J] = v[N2 * J + n2]; });
        RegFft<R, N1, B>::run(a);
        static_for<N1>([&](auto J) {
          constexpr int j = J;
          v[N2 * j + n2] = rot<R, n2 * j, N, B>(a[j]);
        });
      });
      cx<R> out[N];
      static_for<N1>([&](auto J) {
        constexpr int j = J;
        cx<R> a[N2];
        static_for<N2>([&](auto I) { a[I] = v[N2 * j + I]; });
        RegFft<R, N2, B>::run(a);
        static_for<N2>([&](auto I) {
          constexpr int i = I;
          out[j + N1 * i] = a[i];
        });
      });
      static_for<N>([&](auto J) { v[J] = out[J]; });
    }
  }
};
template <typename R, int N, bool B>
__device__ __forceinline__ void reg_fft(cx<R> (&v)[N]) {
  RegFft<R, N, B>::run(v);
}

// longest pencil of one thread: 128 registers of data (t axes split over two
// threads from 32 elements in FP32: 0.079 against 0.066 ms at 32^3 x 64)
template <typename R>
constexpr int kRegMax = sizeof(R) == 8 ? 32 : 64;

// resident blocks asked of the compiler: threads of `data` registers and some
// 44 others, and `smem` bytes a block
__host__ __device__ constexpr int reg_blocks(int threads, int data, size_t smem) {
  const int w = (threads + 31) / 32 * 32;
  int n = 65536 / (w * (data + 44));
  if (smem && n > (int)(220 * 1024 / smem)) n = (int)(220 * 1024 / smem);
  return n < 1 ? 1 : n > 16 ? 16 : n;
}

// --- pencils shared by lanes ------------------------------------------------
// Radix-2 steps between lanes D apart of which h = 0 holds the even and h = 1
// the odd half of an N-point transform, v[i] at some k of N/2 each.  Forward:
// X[k] = E[k] + W^k O[k] and X[k + N/2] = E[k] - W^k O[k] for half of the k, to
// v[j] and v[j + Q]; k = j + h N/4, or j + h8 N/8 + h N/4 after a step before.
template <typename R, int N, int Q, int D>
__device__ __forceinline__ void lane_fwd(cx<R> (&v)[2 * Q], int h, int h8 = 0) {
  static_for<Q>([&](auto J) {
    constexpr int j = J;
    const cx<R> snd = h ? v[j] : v[j + Q];
    const cx<R> rcv = mk<R>(__shfl_xor_sync(0xffffffffu, snd.x, D),
                            __shfl_xor_sync(0xffffffffu, snd.y, D));
    const cx<R> e = h ? rcv : v[j];
    cx<R> o = rot<R, j, N, false>(h ? v[j + Q] : rcv);
    if (h8) o = rot<R, 1, 8, false>(o);
    if (h) o = mk<R>(o.y, -o.x);
    v[j] = cadd(e, o);
    v[j + Q] = csub(e, o);
  });
}
// back: E' = X[k] + X[k + N/2], O' = (X[k] - X[k + N/2]) W^-k
template <typename R, int N, int Q, int D>
__device__ __forceinline__ void lane_bwd(cx<R> (&v)[2 * Q], int h, int h8 = 0) {
  static_for<Q>([&](auto J) {
    constexpr int j = J;
    const cx<R> s = cadd(v[j], v[j + Q]);
    cx<R> d = rot<R, j, N, true>(csub(v[j], v[j + Q]));
    if (h8) d = rot<R, 1, 8, true>(d);
    if (h) d = mk<R>(-d.y, d.x);
    const cx<R> out = h ? s : d;
    const cx<R> in = mk<R>(__shfl_xor_sync(0xffffffffu, out.x, D),
                           __shfl_xor_sync(0xffffffffu, out.y, D));
    v[j] = h ? in : s;
    v[j + Q] = h ? d : in;
  });
}

// --- xy planes of N x N ---------------------------------------------------
// PL planes of one field per block, N threads to each: rows, then columns
// (k_fft_xy is the generic form).  Resident blocks: as many as hold 128
// registers of data and their temporaries.
template <typename R, int N, int PL>
__host__ __device__ constexpr size_t xy_reg_smem() {
  return (size_t)PL * N * (N + 1) * 2 * sizeof(R);
}
template <typename R, int N, int PL, bool B>
__global__ void __launch_bounds__(N *PL, reg_blocks(N *PL, N * sizeof(R) / 2, xy_reg_smem<R, N, PL>()))
    k_fft_xy_reg(Ctx<R> c, int, int prsum) {
  if (xy_done(c, B)) return;
  if (c.skip && c.skip[blockIdx.x / (gridDim.x / c.L[3])]) return;  // finished slice
  extern __shared__ unsigned char smem_raw[];
  constexpr int P = N + 1, T = P * N;
  cx<R> *A = reinterpret_cast<cx<R> *>(smem_raw);
  const int field = blockIdx.y, par = c.st->parity;
  const size_t base = (size_t)field * c.V + (size_t)blockIdx.x * (PL * N * N);
  cx<R> *data = pick(c.fb, par) + base;
  for (int e = threadIdx.x; e < PL * N * N; e += PL * N)
    cp_async(A + (e / N) * P + e % N, data + e);
  cp_async_wait();
  __syncthreads();
  const int pl = threadIdx.x / N, i = threadIdx.x % N;
  cx<R> *tile = A + pl * T;
  cx<R> v[N];
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = tile[i * P + k];
  reg_fft<R, N, B>(v);
#pragma unroll
  for (int k = 0; k < N; k++) tile[i * P + k] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = tile[k * P + i];
  constexpr bool RAG = N * PL % 32 != 0;
  // the previous field, for the sums, on its way into the tile meanwhile
  // (32^3 x 64: 0.087 ms, FP32 0.053; loaded by the sums themselves 0.090 and
  // 0.066, 16^3 x 32 0.015 and 0.013 against 0.019 and 0.016)
  const bool sums = B && prsum;
  if (sums) {
    const cx<R> *old = pick(c.fb, par ^ 1) + base;
    __syncthreads();
    for (int e = threadIdx.x; e < PL * N * N; e += PL * N)
      cp_async(A + (e / N) * P + e % N, old + e);
  }
  reg_fft<R, N, B>(v);
  data += (size_t)pl * N * N + i;
#pragma unroll
  for (int k = 0; k < N; k++) data[k * N] = v[k];
  if (sums) {
    double s[2] = {0.0, 0.0};
    cp_async_wait();
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
      const cx<R> od = tile[k * P + i];
      const double a = v[k].x, b = v[k].y;
      const double tr = a - (double)od.x, ti = b - (double)od.y;
      if (field == 0) {
        s[0] += 2.0 * (a * a + b * b + a * b);
        s[1] += 2.0 * (a * tr + b * ti) + (a * ti + b * tr);
      } else {
        s[0] += 2.0 * (a * a + b * b);
        s[1] += 2.0 * (a * tr + b * ti);
      }
    }
    xy_sums_begin<RAG>(c, s);
    xy_sums<RAG>(c, s);
  }
}

// --- xy planes of N x N, each pencil shared by two lanes --------------------
// For FP64 planes beyond 32: half a pencil fits a thread where a whole one
// doesn't.  Per launch, forward and inverse with sums, before (fft_ct; 36 and
// 40 generic) and now: 36^3 x 72 0.454 + 0.525 -> 0.086 + 0.130 ms, 40^3 x 80
// 0.690 + 0.798 -> 0.115 + 0.174, 48^3 x 96 0.480 + 0.700 -> 0.210 + 0.332 (0.94
// to 0.99 of the copy bandwidth), Coulomb 64^3 x 16 0.174 + 0.249 -> 0.097 +
// 0.139.
template <typename R, int N, int PL, bool B>
__global__ void __launch_bounds__(2 * N *PL, reg_blocks(2 * N *PL, N *sizeof(R) / 4 - 4,
                                                        xy_reg_smem<R, N, PL>()))
    k_fft_xy_pair(Ctx<R> c, int, int prsum) {
  static_assert(N % 4 == 0 && N * PL % 16 == 0, "whole warps");
  if (xy_done(c, B)) return;
  if (c.skip && c.skip[blockIdx.x / (gridDim.x / c.L[3])]) return;  // finished slice
  extern __shared__ unsigned char smem_raw[];
  constexpr int P = N + 1, NT = 2 * N * PL, M = N / 2, Q = M / 2;
  cx<R> *A = reinterpret_cast<cx<R> *>(smem_raw);
  const int field = blockIdx.y, par = c.st->parity;
  const size_t base = (size_t)field * c.V + (size_t)blockIdx.x * (PL * N * N);
  cx<R> *data = pick(c.fb, par) + base;
  for (int e = threadIdx.x; e < PL * N * N; e += NT) cp_async(A + (e / N) * P + e % N, data + e);
  cp_async_wait();
  __syncthreads();
  // lanes 0-15 the even, 16-31 the odd elements of 16 pencils (plane, i); the
  // transform's other side at k = j + h Q and k + M
  const int h = (threadIdx.x >> 4) & 1, q = (threadIdx.x >> 5) * 16 + (threadIdx.x & 15);
  const int pl = q / N, i = q % N;
  cx<R> *tile = A + pl * (P * N);
  auto pos = [&](int n, bool freq) { return freq ? n % Q + n / Q * M + h * Q : 2 * n + h; };
  cx<R> v[M];
  auto fft = [&]() {
    if constexpr (!B) {
      reg_fft<R, M, false>(v);
      lane_fwd<R, N, Q, 16>(v, h);
    } else {
      lane_bwd<R, N, Q, 16>(v, h);
      reg_fft<R, M, true>(v);
    }
  };
#pragma unroll
  for (int n = 0; n < M; n++) v[n] = tile[i * P + pos(n, B)];
  fft();
#pragma unroll
  for (int n = 0; n < M; n++) tile[i * P + pos(n, !B)] = v[n];
  __syncthreads();
#pragma unroll
  for (int n = 0; n < M; n++) v[n] = tile[pos(n, B) * P + i];
  const bool sums = B && prsum;
  if (sums) {
    const cx<R> *old = pick(c.fb, par ^ 1) + base;
    __syncthreads();
    for (int e = threadIdx.x; e < PL * N * N; e += NT) cp_async(A + (e / N) * P + e % N, old + e);
  }
  fft();
  data += (size_t)pl * N * N + i;
#pragma unroll
  for (int n = 0; n < M; n++) data[pos(n, !B) * N] = v[n];
  if (sums) {
    double s[2] = {0.0, 0.0};
    cp_async_wait();
    __syncthreads();
#pragma unroll
    for (int n = 0; n < M; n++) {
      const cx<R> od = tile[pos(n, !B) * P + i];
      const double a = v[n].x, b = v[n].y;
      const double tr = a - (double)od.x, ti = b - (double)od.y;
      if (field == 0) {
        s[0] += 2.0 * (a * a + b * b + a * b);
        s[1] += 2.0 * (a * tr + b * ti) + (a * ti + b * tr);
      } else {
        s[0] += 2.0 * (a * a + b * b);
        s[1] += 2.0 * (a * tr + b * ti);
      }
    }
    xy_sums_begin<false>(c, s);
    xy_sums<false>(c, s);
  }
}

// 1 / p^2 of GLU's gen_p_sq (src/Geometry/geometry.c:169-186) times maxp
template <typename R>
__device__ __forceinline__ R psq_of(double kcos, double D, double maxp) {
  const double p2 = (kcos == D) ? 1.0 : 2.0 * (D - kcos);
  return (R)(maxp * __drcp_rn(p2));
}

// --- z and t of a tile of BW x columns --------------------------------------
template <typename R, int LT>
constexpr bool zt_split = LT > kRegMax<R>;
template <typename R, int LZ, int LT, int BW>
__host__ __device__ constexpr int zt_reg_threads() {
  const int p = LZ * BW;
  return zt_split<R, LT> ? (p + 15) / 16 * 32 : (p + 31) / 32 * 32;
}

template <typename R, int LZ, int LT, int BW>
__host__ __device__ constexpr size_t zt_reg_smem() {
  return (size_t)(LZ * BW + zt_pad(BW)) * LT * 2 * sizeof(R);
}
template <typename R, int LZ, int LT, int BW>
__host__ __device__ constexpr int zt_reg_blocks() {
  const int n = zt_split<R, LT> ? LT / 2 : LT;
  return reg_blocks(zt_reg_threads<R, LZ, LT, BW>(), (n > LZ ? n : LZ) * sizeof(R) / 2,
                    zt_reg_smem<R, LZ, LT, BW>());
}

template <typename R, int LZ, int LT, int BW>
__global__ void __launch_bounds__(zt_reg_threads<R, LZ, LT, BW>(),
                                  zt_reg_blocks<R, LZ, LT, BW>())
    k_fft_zt_reg(Ctx<R> c) {
  if (c.st->done) return;
  constexpr int TS = LZ * BW + zt_pad(BW), NT = zt_reg_threads<R, LZ, LT, BW>();
  constexpr int NPZ = LT * BW, NPT = LZ * BW;
  extern __shared__ unsigned char smem_raw[];
  cx<R> *A = reinterpret_cast<cx<R> *>(smem_raw);
  const int nxb = c.L[0] / BW;
  const int y = blockIdx.x / nxb;
  const size_t sz = (size_t)c.L[0] * c.L[1];
  const int x0 = blockIdx.x % nxb * BW;
  cx<R> *data = pick(c.fb, c.st->parity) + (size_t)blockIdx.y * c.V + (size_t)c.L[0] * y + x0;
  const double cxy = c.cs[c.cs_ld + y];
  const double *cz = c.cs + 2 * c.cs_ld, *ct = c.cs + 3 * c.cs_ld;
#pragma unroll 1
  for (int p = threadIdx.x; p < NPZ; p += NT) {
    const int b = p % BW, t = p / BW;
    const cx<R> *g = data + b + sz * (LZ * t);
    cx<R> v[LZ];
#pragma unroll
    for (int k = 0; k < LZ; k++) v[k] = g[sz * k];
    reg_fft<R, LZ, false>(v);
#pragma unroll
    for (int k = 0; k < LZ; k++) A[b + BW * k + TS * t] = v[k];
  }
  __syncthreads();
  if constexpr (!zt_split<R, LT>) {
    const int p = threadIdx.x;
    if (p < NPT) {
      const double k3 = c.cs[x0 + p % BW] + cxy + cz[p / BW];
      cx<R> v[LT];
#pragma unroll
      for (int t = 0; t < LT; t++) v[t] = A[p + TS * t];
      reg_fft<R, LT, false>(v);
#pragma unroll
      for (int t = 0; t <= LT / 2; t++) {  // psq is even in t
        const R f = psq_of<R>(k3 + ct[t], 4.0, c.maxp);
        v[t] = cscale(v[t], f);
        if (t > 0 && 2 * t < LT) v[LT - t] = cscale(v[LT - t], f);
      }
      reg_fft<R, LT, true>(v);
#pragma unroll
      for (int t = 0; t < LT; t++) A[p + TS * t] = v[t];
    }
  } else {
    // lanes 0-15 the even, 16-31 the odd t of 16 pencils
    constexpr int H = LT / 2, Q = H / 2;
    static_assert(LT % 4 == 0 && H <= kRegMax<R>, "split t axis");
    const int h = (threadIdx.x >> 4) & 1;
    const int p = (threadIdx.x >> 5) * 16 + (threadIdx.x & 15);
    const bool on = p < NPT;
    const int pc = on ? p : 0;
    const double k3 = c.cs[x0 + pc % BW] + cxy + cz[pc / BW];
    cx<R> v[H];
#pragma unroll
    for (int n = 0; n < H; n++) v[n] = A[pc + TS * (2 * n + h)];
    reg_fft<R, H, false>(v);
    // X[k] = E[k] + W^k O[k], X[k + H] = E[k] - W^k O[k] for k = j + h Q
    static_for<Q>([&](auto J) {
      constexpr int j = J;
      const cx<R> snd = h ? v[j] : v[j + Q];
      const cx<R> rcv = mk<R>(__shfl_xor_sync(0xffffffffu, snd.x, 16),
                              __shfl_xor_sync(0xffffffffu, snd.y, 16));
      const cx<R> e = h ? rcv : v[j];
      cx<R> o = rot<R, j, LT, false>(h ? v[j + Q] : rcv);
      if (h) o = mk<R>(o.y, -o.x);  // W^Q = -i
      const R f0 = psq_of<R>(k3 + ct[j + h * Q], 4.0, c.maxp);
      const R f1 = psq_of<R>(k3 + ct[j + h * Q + H], 4.0, c.maxp);
      const cx<R> a = cscale(cadd(e, o), f0), b = cscale(csub(e, o), f1);
      // back: E' = X[k] + X[k + H], O' = (X[k] - X[k + H]) W^-k
      const cx<R> s = cadd(a, b);
      cx<R> d = rot<R, j, LT, true>(csub(a, b));
      if (h) d = mk<R>(-d.y, d.x);
      const cx<R> out = h ? s : d;
      const cx<R> in = mk<R>(__shfl_xor_sync(0xffffffffu, out.x, 16),
                             __shfl_xor_sync(0xffffffffu, out.y, 16));
      v[j] = h ? in : s;
      v[j + Q] = h ? d : in;
    });
    reg_fft<R, H, true>(v);
    if (on) {
#pragma unroll
      for (int n = 0; n < H; n++) A[p + TS * (2 * n + h)] = v[n];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int p = threadIdx.x; p < NPZ; p += NT) {
    const int b = p % BW, t = p / BW;
    cx<R> v[LZ];
#pragma unroll
    for (int k = 0; k < LZ; k++) v[k] = A[b + BW * k + TS * t];
    reg_fft<R, LZ, true>(v);
    cx<R> *g = data + b + sz * (LZ * t);
#pragma unroll
    for (int k = 0; k < LZ; k++) g[sz * k] = v[k];
  }
}

// --- z over two and t over four threads, W of the BW columns at a time ------
// For axes whose pencils leave a thread too few registers or a block too few
// warps: a thread holds a quarter of a t pencil, so that tiles of 32-byte rows
// and twice the warps fit.  Per launch at n^3 x 2n, before (fft_ct, generic
// for 36 and 40; FP32 two threads a t pencil, 2 columns) and now: FP64 48: 1.38
// -> 0.955 ms, 40: 2.00 -> 0.458, 36: 1.13 -> 0.345, 32: 0.162 -> 0.157; FP32
// 48: 0.627 -> 0.492, 40: 0.307 -> 0.229, 36: 0.193 -> 0.155.  Shorter axes lose
// more to the shuffles: FP32 32 0.078 against 0.066 ms, FP64 24 0.044 against
// 0.034, 28 equal.
template <typename R, int LZ, int LT, int W>
__host__ __device__ constexpr int zt_quad_blocks() {
  return reg_blocks(4 * LZ * W, LZ / 2 * sizeof(R) / 2, zt_reg_smem<R, LZ, LT, W>());
}
template <typename R, int LZ, int LT, int BW, int W = BW>
__global__ void __launch_bounds__(4 * LZ * W, zt_quad_blocks<R, LZ, LT, W>())
    k_fft_zt_quad(Ctx<R> c) {
  static_assert(LT == 2 * LZ && LZ % 4 == 0 && LZ * W % 8 == 0, "whole warps");
  if (c.st->done) return;
  constexpr int TS = LZ * W + zt_pad(W), M = LZ / 2, Q = M / 2;
  extern __shared__ unsigned char smem_raw[];
  cx<R> *A = reinterpret_cast<cx<R> *>(smem_raw);
  const int nxb = c.L[0] / BW;
  const int y = blockIdx.x / nxb;
  const size_t sz = (size_t)c.L[0] * c.L[1];
  cx<R> *row = pick(c.fb, c.st->parity) + (size_t)blockIdx.y * c.V + (size_t)c.L[0] * y;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // z: lanes 0-15 the even, 16-31 the odd z of 16 pencils (b, t)
  const int zh = lane >> 4, zp = w * 16 + (lane & 15), zb = zp % W, zt = zp / W;
  cx<R> *const Az = A + zb + TS * zt;
  // t: t = 4 n + 2 h0 + h1 of 8 pencils (b, z)
  const int h0 = (lane >> 3) & 1, h1 = lane >> 4, tp = w * 8 + (lane & 7);
  cx<R> *const At = A + tp + TS * (2 * h0 + h1);
#pragma unroll 1
  for (int sub = 0; sub < BW / W; sub++) {
    const int x0 = blockIdx.x % nxb * BW + sub * W;
    cx<R> *const g = row + x0 + zb + sz * (LZ * zt + zh);
    if (sub) __syncthreads();
    cx<R> v[M];
#pragma unroll
    for (int n = 0; n < M; n++) v[n] = g[sz * (2 * n)];
    reg_fft<R, M, false>(v);
    lane_fwd<R, LZ, Q, 16>(v, zh);
#pragma unroll
    for (int i = 0; i < M; i++) Az[W * (i % Q + i / Q * M + zh * Q)] = v[i];
    __syncthreads();
#pragma unroll
    for (int n = 0; n < M; n++) v[n] = At[TS * 4 * n];
    reg_fft<R, M, false>(v);
    lane_fwd<R, 2 * M, Q, 8>(v, h0);
    lane_fwd<R, 4 * M, Q, 16>(v, h1, h0);
    {
      const double k3 = c.cs[x0 + tp % W] + c.cs[c.cs_ld + y] + c.cs[2 * c.cs_ld + tp / W];
      const double *ct = c.cs + 3 * c.cs_ld + Q * h0 + 2 * Q * h1;
#pragma unroll
      for (int i = 0; i < M; i++) {
        v[i] = cscale(v[i], psq_of<R>(k3 + ct[i % Q + i / Q * (2 * M)], 4.0, c.maxp));
        if (i % 4 == 3) asm volatile("" ::: "memory");  // (not all cosines at once)
      }
    }
    lane_bwd<R, 4 * M, Q, 16>(v, h1, h0);
    lane_bwd<R, 2 * M, Q, 8>(v, h0);
    reg_fft<R, M, true>(v);
#pragma unroll
    for (int n = 0; n < M; n++) At[TS * 4 * n] = v[n];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < M; i++) v[i] = Az[W * (i % Q + i / Q * M + zh * Q)];
    lane_bwd<R, LZ, Q, 16>(v, zh);
    reg_fft<R, M, true>(v);
#pragma unroll
    for (int n = 0; n < M; n++) g[sz * (2 * n)] = v[n];
  }
}

// --- z of Coulomb slices: one pencil per thread, no shared memory ----------
constexpr int kZThreads = 64;

template <typename R, int LZ>
__global__ void __launch_bounds__(kZThreads) k_fft_z_reg(Ctx<R> c) {
  if (c.st->done) return;
  const int n = c.L[0] * c.L[1], nb = (n + kZThreads - 1) / kZThreads;
  const int t = blockIdx.x / nb;
  if (c.skip && c.skip[t]) return;
  const int col = (blockIdx.x % nb) * kZThreads + threadIdx.x;
  if (col >= n) return;
  cx<R> *g = pick(c.fb, c.st->parity) + (size_t)blockIdx.y * c.V + (size_t)t * LZ * n + col;
  const double k2 = c.cs[col % c.L[0]] + c.cs[c.cs_ld + col / c.L[0]];
  const double *cz = c.cs + 2 * c.cs_ld;
  cx<R> v[LZ];
#pragma unroll
  for (int k = 0; k < LZ; k++) v[k] = g[(size_t)k * n];
  reg_fft<R, LZ, false>(v);
#pragma unroll
  for (int k = 0; k <= LZ / 2; k++) {
    const R f = psq_of<R>(k2 + cz[k], 3.0, c.maxp);
    v[k] = cscale(v[k], f);
    if (k > 0 && 2 * k < LZ) v[LZ - k] = cscale(v[LZ - k], f);
  }
  reg_fft<R, LZ, true>(v);
#pragma unroll
  for (int k = 0; k < LZ; k++) g[(size_t)k * n] = v[k];
}

}  // namespace gfix
