// Job descriptors and the variance-to-mean arithmetic of the 1-D bandwidth steps (pkde_steps1d.cu).
#pragma once

#include "pkde_lines.cuh"
#include "pkde_step.cuh"

namespace pkde {

// One estimation (device-resident descriptor).  A tile holds the L = 2 a arrays (z, w) of
// a bootstrap pairs; index 0 / 1 / 2: full tile, last tile, means (L = 1).
struct Job1 {
  int n, npairs, nboot, S, a, P, nst;
  int fused;  // 1: the arithmetic of the step engine's power-of-two tiles, 0: every operation rounded by itself
  int L[3];
  FastDiv dL[3];
  int64_t tab_stride;
  const double2 *spectra;
  const double *fz, *fw, *cw, *vscale;
  double invG, ns, inv_ns;
  double *f_out, *mu_out;
  double2 *state;  // S x n running (mean, m2), lines too long for shared memory
  Stage1 st[kStages1];
};

// x / d correctly rounded for an integer 1 <= d < 2^31 and rd = 1 / d rounded: the residual
// x - q d of the first quotient is exact (an integer multiple of ulp(q) below 2^33 of
// them), and x / d is either representable or at least ulp / (2 d) away from a rounding
// midpoint, far more than the error of the correction.  For x whose exponent field is in
// [100, 2000], where nothing underflows or overflows.
__device__ __forceinline__ double div_int(double x, double d, double rd) {
  const double q = __dmul_rn(x, rd);
  return __fma_rn(__fma_rn(-q, d, x), rd, q);
}

// v / m correctly rounded for m > 0 whose mantissa is not all ones, where nothing leaves the normal
// range: the reciprocal estimate refined to the correctly rounded reciprocal (two iterations
// bring it within an ulp, a third one with the exact remainder rounds it correctly), the quotient
// corrected once by its exact remainder (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990, theorems on the final steps).
__device__ __forceinline__ double div_markstein(double v, double m) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
  y = __fma_rn(y, __fma_rn(-m, y, 1.0), y);
  y = __fma_rn(y, __fma_rn(-m, y, 1.0), y);
  y = __fma_rn(y, __fma_rn(-m, y, 1.0), y);
  const double q = __dmul_rn(v, y);
  return __fma_rn(__fma_rn(-m, q, v), y, q);
}

// VMR of the two bootstraps of a pair at one point (the second one may not exist) and its Welford update
// (DirectSpace.jl:550-552, 572-577), i the first one's number: IEEE divisions.  A call, so that the
// loop around it keeps its registers.
static __device__ __noinline__ double2 vmr_ieee2(double2 z, double2 w, double ns, double i, bool has_b, double2 st) {
  auto add = [&](double Mv, double Vv, double d) {
    const double m = __ddiv_rn(fabs(Mv), ns), a = __ddiv_rn(fabs(Vv), ns);
    const double x = __ddiv_rn(__dsub_rn(a, __dmul_rn(m, m)), m);
    const double delta = __dsub_rn(x, st.x);
    st.x = __dadd_rn(st.x, __ddiv_rn(delta, d));
    st.y = __dadd_rn(st.y, __dmul_rn(delta, __dsub_rn(x, st.x)));
  };
  add(z.x, w.x, i);
  if (has_b) add(z.y, w.y, __dadd_rn(i, 1.0));
  return st;
}

// The same, inv_i = 1 / i and inv_j = 1 / (i + 1).  FUSED: the arithmetic of the step engine's tiles.
// Else every operation rounded by itself, the quotients from products; one range test covers both
// bootstraps, and a mean that is NaN already needs none (see div_nr2).
template <bool FUSED>
__device__ __forceinline__ void vmr_update2(double2 z, double2 w, double ns, double inv_ns, double i, double inv_i,
                                            double inv_j, bool has_b, double2 &st) {
  if constexpr (FUSED) {
    const double ma = __dmul_rn(fabs(z.x), inv_ns), mb = __dmul_rn(fabs(z.y), inv_ns);
    double xa, xb;
    div_nr2(__fma_rn(fabs(w.x), inv_ns, -__dmul_rn(ma, ma)), ma, __fma_rn(fabs(w.y), inv_ns, -__dmul_rn(mb, mb)), mb,
            st.x, xa, xb);
    auto add = [&st](double x, double inv) {
      const double delta = __dsub_rn(x, st.x);
      st.x = __fma_rn(delta, inv, st.x);
      st.y = __fma_rn(delta, __dsub_rn(x, st.x), st.y);
    };
    add(xa, inv_i);
    if (has_b) add(xb, inv_j);
  } else {
    // below 1401 << 21 where the exponent field is in [300, 1700]
    auto range_of = [](double x) { return 2u * (unsigned)__double2hiint(x) - (300u << 21); };
    double2 t = st;
    unsigned range = 0;
    auto add = [&](double Mv, double Vv, double d, double rd) {
      const double m = div_int(fabs(Mv), ns, inv_ns), a = div_int(fabs(Vv), ns, inv_ns);
      const double v = __dsub_rn(a, __dmul_rn(m, m));
      const double x = div_markstein(v, m);
      const double delta = __dsub_rn(x, t.x);
      const unsigned ones = (unsigned)__double2loint(m) == 0xffffffffu ? 0xffffffffu : 0u;
      range = max(max(max(range, range_of(Mv)), max(range_of(Vv), range_of(v))), max(range_of(delta), ones));
      t.x = __dadd_rn(t.x, div_int(delta, d, rd));
      t.y = __dadd_rn(t.y, __dmul_rn(delta, __dsub_rn(x, t.x)));
    };
    add(z.x, w.x, i, inv_i);
    if (has_b) add(z.y, w.y, __dadd_rn(i, 1.0), inv_j);
    if (range >= 1401u << 21) {
      if (!isnan(st.x)) t = vmr_ieee2(z, w, ns, i, has_b, st);
    }
    st = t;
  }
}

// The steps of `count` jobs of one 2^a 3^b 5^c length with a kernel of its own (pkde_steps1d_len.cuh).
bool steps1d_len_known(int n);
void steps1d_len_run(pkde_ctx *ctx, int n, const Job1 *jobs, int count, int S, cudaStream_t st);

}  // namespace pkde
