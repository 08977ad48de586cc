// Stockham FFT stages over tiles of lines of any length, several lines a tile (element k
// of line l at unit k P + l: lanes run over lines, then butterflies, so that accesses are
// contiguous and the lines of a butterfly share one twiddle load).  The arithmetic is that
// of smem_fft (pkde_internal.cuh), operation for operation.
#pragma once

#include "pkde_internal.cuh"

namespace pkde {

constexpr int kStages1 = 8;  // enough for every n <= 4096 (3^7 has seven)

// Stockham stage of radix R: nb = n / R butterflies a line, Ns the product of the earlier
// radices.  tw: twiddles W^(r k) as [k][r - 1] (radix 2, 3, 4, 5, 8), the plain table
// (cos, sin)(2 pi m / n) for other radices.
struct Stage1 {
  int R, nb, Ns, tstep;
  FastDiv dns;
  const double2 *tw;
};

// The transforms' complex product with its fusions written out: the decisions at
// rounding-decided grid points follow the last bit, so a product must not depend on how
// the compiler contracts it in one place or another.
__device__ __forceinline__ double2 cmul1(double2 a, double2 b) {
  return make_double2(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y)));
}

// First level of a radix-8 butterfly on inputs scaled by s: the scaling of one operand of
// each sum is fused into it, as in the register tiles, where the scaled values feed the
// sums directly.
__device__ __forceinline__ void dft4_scaled(double2 *v, const double *s) {
  auto add = [](double a, double sa, double b, double sb) { return __fma_rn(a, sa, __dmul_rn(b, sb)); };
  auto sub = [](double a, double sa, double b, double sb) { return __fma_rn(a, sa, -__dmul_rn(b, sb)); };
  const double2 t0 = make_double2(add(v[0].x, s[0], v[2].x, s[2]), add(v[0].y, s[0], v[2].y, s[2]));
  const double2 t1 = make_double2(sub(v[0].x, s[0], v[2].x, s[2]), sub(v[0].y, s[0], v[2].y, s[2]));
  const double2 t2 = make_double2(add(v[1].x, s[1], v[3].x, s[3]), add(v[1].y, s[1], v[3].y, s[3]));
  const double2 d3 = make_double2(sub(v[1].x, s[1], v[3].x, s[3]), sub(v[1].y, s[1], v[3].y, s[3]));
  const double2 t3 = cmul_si(d3, 1);
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  v[1] = cadd(t1, t3);
  v[3] = csub(t1, t3);
}
// Second level of the radix-8 butterfly from its even and odd halves.
__device__ __forceinline__ void dft8_join(double2 *v, const double2 *e, const double2 *o) {
  const double h = 0.70710678118654752440;  // sqrt(1/2)
  auto join = [h](double2 e, double ax, double ay, double2 &p, double2 &m) {
    p = make_double2(__fma_rn(h, ax, e.x), __fma_rn(h, ay, e.y));
    m = make_double2(__fma_rn(-h, ax, e.x), __fma_rn(-h, ay, e.y));
  };
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  join(e[1], o[1].x - o[1].y, o[1].y + o[1].x, v[1], v[5]);
  const double2 o2 = cmul_si(o[2], 1);
  v[2] = cadd(e[2], o2);
  v[6] = csub(e[2], o2);
  join(e[3], -o[3].x - o[3].y, o[3].x - o[3].y, v[3], v[7]);
}
__device__ __forceinline__ void dft8_scaled(double2 *v, const double *s) {
  double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
  const double se[4] = {s[0], s[2], s[4], s[6]}, so[4] = {s[1], s[3], s[5], s[7]};
  dft4_scaled(e, se);
  dft4_scaled(o, so);
  dft8_join(v, e, o);
}
__device__ __forceinline__ void dft3_fused(double2 *v) {
  const double s3 = 0.86602540378443864676;  // sin(2 pi / 3)
  const double2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
  const double2 m = make_double2(__fma_rn(-0.5, t.x, v[0].x), __fma_rn(-0.5, t.y, v[0].y));
  v[0] = cadd(v[0], t);
  v[1] = make_double2(__fma_rn(-s3, d.y, m.x), __fma_rn(s3, d.x, m.y));
  v[2] = make_double2(__fma_rn(s3, d.y, m.x), __fma_rn(-s3, d.x, m.y));
}
__device__ __forceinline__ void dft5_fused(double2 *v) {
  const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;  // cos(2 pi / 5), cos(4 pi / 5)
  const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;   // sin(2 pi / 5), sin(4 pi / 5)
  const double2 a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
  const double2 a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
  const double2 x0 = v[0];
  auto even = [](double x, double p, double a, double q, double b) { return __fma_rn(q, b, __fma_rn(p, a, x)); };
  auto odd = [](double p, double a, double q, double b) { return __fma_rn(p, a, __dmul_rn(q, b)); };
  const double2 p1 = make_double2(even(x0.x, c1, a1.x, c2, a2.x), even(x0.y, c1, a1.y, c2, a2.y));
  const double2 p2 = make_double2(even(x0.x, c2, a1.x, c1, a2.x), even(x0.y, c2, a1.y, c1, a2.y));
  const double2 q1 = cmul_si(make_double2(odd(s1, b1.x, s2, b2.x), odd(s1, b1.y, s2, b2.y)), 1);
  const double2 q2 = cmul_si(make_double2(odd(s2, b1.x, -s1, b2.x), odd(s2, b1.y, -s1, b2.y)), 1);
  v[0] = cadd(x0, cadd(a1, a2));
  v[1] = cadd(p1, q1);
  v[4] = csub(p1, q1);
  v[2] = cadd(p2, q2);
  v[3] = csub(p2, q2);
}
template <int R>
__device__ __forceinline__ void dft_r(double2 *v) {
  if constexpr (R == 2) dft2<1>(v);
  if constexpr (R == 3) dft3_fused(v);
  if constexpr (R == 4) dft4<1>(v);
  if constexpr (R == 5) dft5_fused(v);
  if constexpr (R == 8) {
    double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4<1>(e);
    dft4<1>(o);
    dft8_join(v, e, o);
  }
}

// Any other radix: an item is four outputs of one butterfly of two lines, l and l + H (2 H lines
// of which L exist).  tw(o): the factor at byte o of the plain table; ld(p): the element at p,
// input r of butterfly j of line l at p = (j + r nb) PB + 16 l; st(l, pos, v): output pos of line l.
// Six FP64 operations a term, two issue slots each; the two lines share the loads of the
// factors and their index steps, which else fill the rest of the slots and the load pipe.  The 41
// points of 50 x 41 x 36, 32 bootstraps, 100 steps: 8.5 ms from the L1 with an item a line, 7.1 with the
// factors in shared memory, 6.5 here (67 % of the FP64 pipe); the 77 of 150 x 77: 5.3, 5.1, 4.4.
template <int T, class Tw, class Ld, class St>
__device__ __forceinline__ void line_stage_generic(const Stage1 &s, int n, int L, int H, FastDiv dH, unsigned PB, Tw tw,
                                                   Ld ld, St st) {
  constexpr int QB = 4;
  const int R = s.R, nb = s.nb, Ns = s.Ns;
  const int nblk = (R + QB - 1) / QB, per = nb * H;
  const unsigned end = n * 16u, d = nb * PB;
  for (int i = threadIdx.x; i < nblk * per; i += T) {
    const int qb = i / per, e = i - qb * per;
    const int j = (int)fdiv((uint32_t)e, dH), l = e - j * H;
    const int jq = (int)fdiv((uint32_t)j, s.dns), k = j - jq * Ns;
    const int q0 = qb * QB, nq = min(QB, R - q0);
    const bool two = l + H < L;
    double2 v[QB], w[QB];
    unsigned m[QB], inc[QB];
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      m[q] = 0;
      inc[q] = q < nq ? (unsigned)(k * s.tstep + (q0 + q) * nb) * 16u : 0;
      v[q] = w[q] = make_double2(0.0, 0.0);
    }
    unsigned p = j * PB + l * 16u;
    const unsigned next = two ? H * 16u : 0;
#pragma unroll 1
    for (int r = 0; r < R; ++r, p += d) {
      const double2 x = ld(p), y = ld(p + next);
#pragma unroll
      for (int q = 0; q < QB; ++q) {
        const double2 f = tw(m[q]);
        v[q] = cadd(v[q], cmul1(x, f));
        w[q] = cadd(w[q], cmul1(y, f));
        const unsigned t = m[q] + inc[q];
        m[q] = min(t, t - end);
      }
    }
    const int o = j + jq * Ns * (R - 1) + q0 * Ns;
#pragma unroll
    for (int q = 0; q < QB; ++q)
      if (q < nq) {
        st(l, o + q * Ns, v[q]);
        if (two) st(l + H, o + q * Ns, w[q]);
      }
  }
}

// Host: the stages of an n-point line (radix sequence of make_plan, tables on the device);
// returns their number.
bool stages_ok(int n);
int make_stages(pkde_ctx *ctx, int n, Stage1 *stages, cudaStream_t st);

}  // namespace pkde
