// SU(3) algebra for the gauge-fixing kernels, templated on the working
// precision R (double or float).  Matrices are 9 complex numbers in
// row-major order, the layout of GLU's lat[i].O[mu].
//
// The operations reproduce the reference's SSE code paths, which are what a
// default x86 build of GLU executes:
//   gram_reunit        column Gram-Schmidt, column 2 = conj(col0 x col1)
//                      (src/Matrix_Ops/gramschmidt_SSE.c:37-98)
//   set_gauge_matrix   g = reunit(1 + alpha A) from the packed fields,
//                      only columns 0 and 1 filled (src/Gfix/CG.c:72-97)
//   gtransform         b <- a b c^dag, columns 0,1 explicit, column 2 by
//                      conj cross product (src/Gfix/gtrans.c:31-141)
//   probe_trace        Re tr(a b c^dag) (src/Matrix_Ops/trace_abc_SSE.c:34-114)
//                      of the line search, c = reunit(1 + alpha A) not formed
//   multab             a <- b c, row 2 by cross product
//                      (src/Matrix_Ops/MMUL/MMUL_SUNC_SSE.c:30-76)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gfix {

template <typename R>
struct alignas(2 * sizeof(R)) cx {
  R x, y;
};

template <typename R>
__host__ __device__ __forceinline__ cx<R> mk(R a, R b) {
  cx<R> r;
  r.x = a;
  r.y = b;
  return r;
}

// a*b in the FMA form of the reference's SSE2_MUL
template <typename R>
__device__ __forceinline__ cx<R> cmul(cx<R> a, cx<R> b) {
  return mk<R>(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// a*conj(b)
template <typename R>
__device__ __forceinline__ cx<R> cmulc(cx<R> a, cx<R> b) {
  return mk<R>(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -(a.x * b.y)));
}
// conj(a)*b
template <typename R>
__device__ __forceinline__ cx<R> ccmul(cx<R> a, cx<R> b) {
  return mk<R>(fma(a.x, b.x, a.y * b.y), fma(a.x, b.y, -(a.y * b.x)));
}
template <typename R>
__device__ __forceinline__ cx<R> cadd(cx<R> a, cx<R> b) {
  return mk<R>(a.x + b.x, a.y + b.y);
}
template <typename R>
__device__ __forceinline__ cx<R> csub(cx<R> a, cx<R> b) {
  return mk<R>(a.x - b.x, a.y - b.y);
}
template <typename R>
__device__ __forceinline__ cx<R> conjg(cx<R> a) {
  return mk<R>(a.x, -a.y);
}
template <typename R>
__device__ __forceinline__ cx<R> cscale(cx<R> a, R s) {
  return mk<R>(a.x * s, a.y * s);
}

// an element fetched to shared memory while the thread goes on (16 or 8
// bytes), and the wait for all that this thread has under way
template <typename R>
__device__ __forceinline__ void cp_async(cx<R> *dst, const cx<R> *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(R) == 8)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// column Gram-Schmidt of columns 0 (u0,u3,u6) and 1 (u1,u4,u7); column 2
// from their conjugate cross product.  The normalisations use rsqrt (within
// an ulp of GLU's 1/sqrt, far cheaper than a division and a square root).
template <typename R>
__device__ __forceinline__ void gram_reunit(cx<R> *u) {
  R n = (u[0].x * u[0].x + u[3].x * u[3].x + u[6].x * u[6].x) +
        (u[0].y * u[0].y + u[3].y * u[3].y + u[6].y * u[6].y);
  R s = rsqrt(n);
  u[0] = cscale(u[0], s);
  u[3] = cscale(u[3], s);
  u[6] = cscale(u[6], s);
  cx<R> p = cadd(cadd(cmulc(u[1], u[0]), cmulc(u[4], u[3])), cmulc(u[7], u[6]));
  u[1] = csub(u[1], cmul(p, u[0]));
  u[4] = csub(u[4], cmul(p, u[3]));
  u[7] = csub(u[7], cmul(p, u[6]));
  n = (u[1].x * u[1].x + u[4].x * u[4].x + u[7].x * u[7].x) +
      (u[1].y * u[1].y + u[4].y * u[4].y + u[7].y * u[7].y);
  s = rsqrt(n);
  u[1] = cscale(u[1], s);
  u[4] = cscale(u[4], s);
  u[7] = cscale(u[7], s);
  u[2] = conjg(csub(cmul(u[3], u[7]), cmul(u[4], u[6])));
  u[5] = conjg(csub(cmul(u[1], u[6]), cmul(u[0], u[7])));
  u[8] = conjg(csub(cmul(u[0], u[4]), cmul(u[1], u[3])));
}

// g = reunit(1 + alpha A) with A from the packed su(3) fields f0..f3
// (GLU's SU(3) packing: f0 = -D1 + i D0, f1, f2, f3 the off-diagonals)
template <typename R>
__device__ __forceinline__ void set_gauge(cx<R> *g, cx<R> f0, cx<R> f1,
                                          cx<R> f2, cx<R> f3, R alpha) {
  g[0] = mk<R>(R(1), alpha * f0.y);
  g[1] = cscale(f1, alpha);
  g[3] = mk<R>(-g[1].x, g[1].y);
  g[4] = mk<R>(R(1), -alpha * f0.x);
  g[6] = mk<R>(-alpha * f2.x, alpha * f2.y);
  g[7] = mk<R>(-alpha * f3.x, alpha * f3.y);
  gram_reunit(g);
}

// the third column of a matrix whose first two columns are set: the
// conjugate cross product of the first two, the completion of gtransform
// (src/Gfix/gtrans.c:107-121) and of gram_reunit
template <typename R>
__device__ __forceinline__ void complete_col2(cx<R> *u) {
  u[2] = conjg(csub(cmul(u[3], u[7]), cmul(u[4], u[6])));
  u[5] = conjg(csub(cmul(u[1], u[6]), cmul(u[0], u[7])));
  u[8] = conjg(csub(cmul(u[0], u[4]), cmul(u[1], u[3])));
}

// b <- a b c^dag
template <typename R>
__device__ __forceinline__ void gtransform(const cx<R> *a, cx<R> *b,
                                           const cx<R> *c) {
  // bc[r][k] = sum_j b[r][j] conj(c[k][j]), k = 0, 1
  cx<R> bc[6];
#pragma unroll
  for (int r = 0; r < 3; r++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      bc[r * 2 + k] = cadd(cadd(cmulc(b[r * 3 + 0], c[k * 3 + 0]),
                                cmulc(b[r * 3 + 1], c[k * 3 + 1])),
                           cmulc(b[r * 3 + 2], c[k * 3 + 2]));
    }
  }
#pragma unroll
  for (int r = 0; r < 3; r++) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      b[r * 3 + k] = cadd(cadd(cmul(a[r * 3 + 0], bc[0 * 2 + k]),
                               cmul(a[r * 3 + 1], bc[1 * 2 + k])),
                          cmul(a[r * 3 + 2], bc[2 * 2 + k]));
    }
  }
  complete_col2(b);
}

// acc + a b, four fused operations
template <typename R>
__device__ __forceinline__ cx<R> cmadd(cx<R> acc, cx<R> a, cx<R> b) {
  return mk<R>(fma(-a.y, b.y, fma(a.x, b.x, acc.x)),
               fma(a.y, b.x, fma(a.x, b.y, acc.y)));
}
// acc + a conj(b)
template <typename R>
__device__ __forceinline__ cx<R> cmaddc(cx<R> acc, cx<R> a, cx<R> b) {
  return mk<R>(fma(a.y, b.y, fma(a.x, b.x, acc.x)),
               fma(-a.x, b.y, fma(a.y, b.x, acc.y)));
}
// conj(a b - c d)
template <typename R>
__device__ __forceinline__ cx<R> cdet(cx<R> a, cx<R> b, cx<R> c, cx<R> d) {
  return mk<R>(fma(c.y, d.y, fma(-c.x, d.x, fma(-a.y, b.y, a.x * b.x))),
               fma(c.y, d.x, fma(c.x, d.y, fma(-a.y, b.x, -(a.x * b.y)))));
}
// x = m v, m a row-major 3x3 matrix
template <typename R>
__device__ __forceinline__ void mat_vec(cx<R> *x, const cx<R> *m, const cx<R> *v) {
#pragma unroll
  for (int r = 0; r < 3; r++)
    x[r] = cmadd(cmadd(cmul(m[3 * r], v[0]), m[3 * r + 1], v[1]), m[3 * r + 2], v[2]);
}

// The line-search traces Re tr(g(x) U g(y)^dag), g = reunit(1 + alpha A),
// without forming g(y).  With a0, a1 the first two columns of A(y) and
// m_j = e_j + alpha a_j, the Gram-Schmidt columns of g(y) are
//   s0 m0,  s1 (m1 - q m0),  s0 s1 conj(m0 x m1),
// and because A is anti-Hermitian, m_i^dag m_j = delta_ij + alpha^2 a_i^dag
// a_j: the norms and the projection q need three inner products and the
// third column one cross product a0 x a1, none of which depends on alpha,
// so both probes of a link share them.  With x_j = g(x) u_j of the first two
// columns of U (the third is conj(x0 x x1)), the trace is
//   s0 Re<m0, x0> + s1 Re(<m1, x1> - conj(q) <m0, x1>)
//     + s0 s1 Re((m0 x m1) . x2),
// 1/s0^2 = 1 + alpha^2 |a0|^2 and 1/(s0 s1)^2 = |m0 x m1|^2 = 1 + alpha^2
// (|a0|^2 + |a1|^2) + alpha^4 |a0 x a1|^2, sums of positive terms.
// About 170 operations per probe against 270 for g(y), the third column of U
// and the product (src/Gfix/line_search.c:274-341 forms them all); the
// matrix 1 + alpha A of the packed fields is that of set_gauge.
template <typename R>
struct ProbeDir {
  R a, b;            // a1_1 = -i a, a0_0 = i b
  cx<R> f1, f2, f3;  // a0 = (i b, -f1*, -f2*), a1 = (f1, -i a, -f3*)
  R h00, hs, nn;     // |a0|^2, |a0|^2 + |a1|^2, |a0 x a1|^2
  cx<R> h01, n0, n1; // <a0, a1>; a0 x a1 = (n0, n1, n2)
  R n2;
};

template <typename R>
__device__ __forceinline__ ProbeDir<R> probe_dir(cx<R> f0, cx<R> f1, cx<R> f2,
                                                 cx<R> f3) {
  ProbeDir<R> p;
  p.a = f0.x;
  p.b = f0.y;
  p.f1 = f1;
  p.f2 = f2;
  p.f3 = f3;
  const R n1 = fma(f1.y, f1.y, f1.x * f1.x);
  p.h00 = fma(f2.y, f2.y, fma(f2.x, f2.x, fma(p.b, p.b, n1)));
  p.hs = p.h00 + fma(f3.y, f3.y, fma(f3.x, f3.x, fma(p.a, p.a, n1)));
  const R d = p.a - p.b;
  p.h01 = cmaddc(mk<R>(-(d * f1.y), d * f1.x), f2, f3);
  // f1* f3* - i a f2*, -f2* f1 + i b f3*, a b + |f1|^2
  p.n0 = mk<R>(fma(-f1.y, f3.y, fma(f1.x, f3.x, -(p.a * f2.y))),
               -fma(f1.y, f3.x, fma(f1.x, f3.y, p.a * f2.x)));
  p.n1 = mk<R>(fma(p.b, f3.y, -fma(f2.y, f1.y, f2.x * f1.x)),
               fma(p.b, f3.x, fma(f2.y, f1.x, -(f2.x * f1.y))));
  p.n2 = fma(p.a, p.b, n1);
  p.nn = fma(p.n0.x, p.n0.x, fma(p.n0.y, p.n0.y, fma(p.n1.x, p.n1.x,
         fma(p.n1.y, p.n1.y, p.n2 * p.n2))));
  return p;
}

// Re tr(A U B^dag) with A = g(x), u0 and u1 the first two columns of U and
// B = g(y) of the direction p at step al
template <typename R>
__device__ __forceinline__ R probe_trace(const cx<R> *A, const cx<R> *u0,
                                         const cx<R> *u1, const ProbeDir<R> &p, R al) {
  cx<R> x0[3], x1[3], x2[3];
  mat_vec(x0, A, u0);
  mat_vec(x1, A, u1);
  x2[0] = cdet(x0[1], x1[2], x0[2], x1[1]);
  x2[1] = cdet(x0[2], x1[0], x0[0], x1[2]);
  x2[2] = cdet(x0[0], x1[1], x0[1], x1[0]);
  const R a2 = al * al;
  const R u = fma(a2, p.h00, R(1));
  const R s0 = rsqrt(u), s01 = rsqrt(fma(a2, fma(a2, p.nn, p.hs), R(1)));
  const R s1 = u * s0 * s01, t = a2 * s0 * s0;
  const cx<R> q = mk<R>(t * p.h01.x, t * p.h01.y);
  // Re<a0, x0>, <a0, x1>, Re<a1, x1>
  const R t0 = fma(p.b, x0[0].y,
                   -fma(p.f1.x, x0[1].x,
                        fma(-p.f1.y, x0[1].y, fma(p.f2.x, x0[2].x, -(p.f2.y * x0[2].y)))));
  cx<R> w = cmadd(cmul(p.f1, x1[1]), p.f2, x1[2]);
  w = mk<R>(fma(p.b, x1[0].y, -w.x), fma(-p.b, x1[0].x, -w.y));
  const R t1 = fma(p.f1.x, x1[0].x,
                   fma(p.f1.y, x1[0].y,
                       -fma(p.a, x1[1].y, fma(p.f3.x, x1[2].x, -(p.f3.y * x1[2].y)))));
  const cx<R> c = mk<R>(fma(al, w.x, x1[0].x), fma(al, w.y, x1[0].y));
  const R T0 = fma(al, t0, x0[0].x);
  const R T1 = fma(-q.y, c.y, fma(-q.x, c.x, fma(al, t1, x1[1].x)));
  // (a0 x e1 + e0 x a1) + al a0 x a1 = (f2*, f3*, i (b - a)) + al (n0, n1, n2)
  const R v0x = fma(al, p.n0.x, p.f2.x), v0y = fma(al, p.n0.y, -p.f2.y);
  const R v1x = fma(al, p.n1.x, p.f3.x), v1y = fma(al, p.n1.y, -p.f3.y);
  const R v2x = al * p.n2, v2y = p.b - p.a;
  R z = fma(v0x, x2[0].x, -(v0y * x2[0].y));
  z = fma(v1x, x2[1].x, fma(-v1y, x2[1].y, z));
  z = fma(v2x, x2[2].x, fma(-v2y, x2[2].y, z));
  const R T2 = fma(al, z, x2[2].x);
  return fma(s0, T0, fma(s1, T1, s01 * T2));
}

// Re tr of an SU(3) matrix given by its first two columns
template <typename R>
__device__ __forceinline__ R re_tr_cols(const cx<R> *u0, const cx<R> *u1) {
  const R c = fma(u0[1].y, u1[0].y, fma(-u0[1].x, u1[0].x,
                  fma(-u0[0].y, u1[1].y, u0[0].x * u1[1].x)));
  return u0[0].x + u1[1].x + c;
}

// a <- b c, row 2 by conj cross product of rows 0 and 1
template <typename R>
__device__ __forceinline__ void multab(cx<R> *a, const cx<R> *b,
                                       const cx<R> *c) {
#pragma unroll
  for (int r = 0; r < 2; r++) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      a[r * 3 + k] = cadd(cmul(b[r * 3 + 0], c[k]),
                          cadd(cmul(b[r * 3 + 1], c[3 + k]),
                               cmul(b[r * 3 + 2], c[6 + k])));
    }
  }
  a[6] = conjg(csub(cmul(a[1], a[5]), cmul(a[2], a[4])));
  a[7] = conjg(csub(cmul(a[2], a[3]), cmul(a[0], a[5])));
  a[8] = conjg(csub(cmul(a[0], a[4]), cmul(a[1], a[3])));
}

// short Hermitian projection of U (src/Matrix_Ops/exactQ.c:400-428):
// q0, q3 real diagonals; q1, q2, q4 the upper off-diagonals
template <typename R>
__device__ __forceinline__ void herm_short(const cx<R> *U, R &q0, cx<R> &q1,
                                           cx<R> &q2, R &q3, cx<R> &q4) {
  const R i0 = U[0].y, i4 = U[4].y, i8 = U[8].y;
  q0 = (R(2) * i0 - i4 - i8) / R(3);
  q3 = (R(2) * i4 - i0 - i8) / R(3);
  // i/2 (conj(U3) - U1) = 0.5 (U3.y + U1.y) + i 0.5 (U3.x - U1.x)
  q1 = mk<R>(R(0.5) * (U[3].y + U[1].y), R(0.5) * (U[3].x - U[1].x));
  q2 = mk<R>(R(0.5) * (U[6].y + U[2].y), R(0.5) * (U[6].x - U[2].x));
  q4 = mk<R>(R(0.5) * (U[7].y + U[5].y), R(0.5) * (U[7].x - U[5].x));
}

template <typename R>
__device__ __forceinline__ void set_identity(cx<R> *u) {
#pragma unroll
  for (int k = 0; k < 9; k++) u[k] = mk<R>(R(0), R(0));
  u[0] = u[4] = u[8] = mk<R>(R(1), R(0));
}

}  // namespace gfix
