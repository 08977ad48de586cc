// Bandwidth steps of 1-D estimations on grids of any length up to 4096: one CTA per step
// (the steps are independent given the spectra) runs the step's bootstrap pairs and the
// full-sample means without leaving the SM.
//
// Reference: GradeProEstimator.jl:968-1051 (the step loop), FourierSpace.jl:215-262
// (propagation), :445-524 (inverse transforms), DirectSpace.jl:526-584 (VMR), :747-764
// (means), :829-1031 (convergence).
//
// The convergence state machine needs a point's steps in order, so the kernel stores each
// step's log scaled variance f_s and means mu_s, and converge_steps_kernel walks them.
#include <algorithm>

#include "pkde_lines.cuh"
#include "pkde_regfft.cuh"
#include "pkde_steps1d.cuh"

namespace pkde {
namespace {

extern __shared__ double2 sm1[];

// A stage over the L lines of a tile, from the tile at unit `src` to the one at `dst`:
// element k of line l at unit k L + l, so that lanes run over lines, then butterflies
// (contiguous reads, one twiddle load for the lines of a butterfly).  P: pitch of the
// written tile.  FIRST: the inputs come from the spectra (line l at in + l n), times the
// step's factors (f0: even lines, f1: odd lines, c0, c1 their scalars).
template <int T, int R, bool FIRST>
__device__ __forceinline__ void stage1(const Stage1 &s, int src, int dst, int n, int L, FastDiv dL, int P,
                                       const double2 *in, const double *f0, const double *f1, double c0, double c1,
                                       int fused) {
  const int nb = s.nb, Ns = FIRST ? 1 : s.Ns, items = nb * L, rs = nb * L, ws = Ns * P;
  const double2 *tw = s.tw;
  const FastDiv dns = s.dns;
  for (int e = threadIdx.x; e < items; e += T) {
    const int j = (int)fdiv((uint32_t)e, dL), l = e - j * L;
    double2 v[R];
    int o;
    if constexpr (FIRST) {
      o = dst + j * R * P + l;
      const double2 *p = in + l * n + j;
      const double *f = ((l & 1) ? f1 : f0) + j;
      const double c = (l & 1) ? c1 : c0;
      double sc[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[r] = __ldg(p + r * nb);
        sc[r] = c * __ldg(f + r * nb);
      }
      bool done = false;
      if constexpr (R == 8) {
        if (fused) {
          dft8_scaled(v, sc);
          done = true;
        }
      }
      if (!done) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = make_double2(__dmul_rn(v[r].x, sc[r]), __dmul_rn(v[r].y, sc[r]));
        dft_r<R>(v);
      }
    } else {
      const int jq = (int)fdiv((uint32_t)j, dns), k = j - jq * Ns;
      o = dst + (j + jq * Ns * (R - 1)) * P + l;
      const double2 *p = sm1 + src + e;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * rs];
      if (k > 0) {
        const double2 *w = tw + k * (R - 1) - 1;
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul1(v[r], __ldg(w + r));
      }
      dft_r<R>(v);
    }
    double2 *q = sm1 + o;
#pragma unroll
    for (int r = 0; r < R; ++r) q[r * ws] = v[r];
  }
}

// Any other radix: an item is QB outputs of one butterfly, every input is read once an item.
template <int T>
__device__ __noinline__ void stage1_generic(const Stage1 &s, int src, int dst, int n, int L, FastDiv dL, int P) {
  constexpr int QB = 4;
  const int R = s.R, nb = s.nb, Ns = s.Ns;
  const int nblk = (R + QB - 1) / QB, per = nb * L;
  for (int i = threadIdx.x; i < nblk * per; i += T) {
    const int qb = i / per, e = i - qb * per;
    const int j = (int)fdiv((uint32_t)e, dL), l = e - j * L;
    const int jq = (int)fdiv((uint32_t)j, s.dns), k = j - jq * Ns;
    const int q0 = qb * QB, nq = min(QB, R - q0);
    double2 v[QB];
    int m[QB], inc[QB];
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      m[q] = 0;
      inc[q] = q < nq ? k * s.tstep + (q0 + q) * nb : 0;
      v[q] = make_double2(0.0, 0.0);
    }
    const double2 *p = sm1 + src + e;
    for (int r = 0; r < R; ++r, p += per) {
      const double2 x = *p;
#pragma unroll
      for (int q = 0; q < QB; ++q) {
        v[q] = cadd(v[q], cmul1(x, __ldg(s.tw + m[q])));
        m[q] += inc[q];
        if (m[q] >= n) m[q] -= n;
      }
    }
    double2 *o = sm1 + dst + (j + jq * Ns * (R - 1) + q0 * Ns) * P + l;
#pragma unroll
    for (int q = 0; q < QB; ++q)
      if (q < nq) o[q * Ns * P] = v[q];
  }
}

// Inverse transform of the L lines at `in`, scaled by the step's factors, through the two
// tiles at units a and b; returns the tile of the results, element k of line l at unit
// k P + l.
template <int T>
__device__ __forceinline__ int transform1(const Job1 &J, int a, int b, const double2 *in, int L, FastDiv dL, int P,
                                          const double *f0, const double *f1, double c0, double c1) {
  const int n = J.n;
  int st = 0, src = a, dst = b;
  {
    const Stage1 &s = J.st[0];
    const int Pw = J.nst == 1 ? P : L;
    switch (s.R) {
      case 8: stage1<T, 8, true>(s, 0, dst, n, L, dL, Pw, in, f0, f1, c0, c1, J.fused); st = 1; break;
      case 4: stage1<T, 4, true>(s, 0, dst, n, L, dL, Pw, in, f0, f1, c0, c1, 0); st = 1; break;
      case 2: stage1<T, 2, true>(s, 0, dst, n, L, dL, Pw, in, f0, f1, c0, c1, 0); st = 1; break;
      case 3: stage1<T, 3, true>(s, 0, dst, n, L, dL, Pw, in, f0, f1, c0, c1, 0); st = 1; break;
      case 5: stage1<T, 5, true>(s, 0, dst, n, L, dL, Pw, in, f0, f1, c0, c1, 0); st = 1; break;
      default:  // a generic radix first: its inputs pass through the tile
        for (int e = threadIdx.x; e < n * L; e += T) {
          const int k = (int)fdiv((uint32_t)e, dL), l = e - k * L;
          const double sc = ((l & 1) ? c1 : c0) * __ldg(((l & 1) ? f1 : f0) + k);
          const double2 x = __ldg(in + l * n + k);
          sm1[dst + e] = make_double2(__dmul_rn(x.x, sc), __dmul_rn(x.y, sc));
        }
    }
    __syncthreads();
  }
  for (; st < J.nst; ++st) {
    const int t = src;
    src = dst;
    dst = t;
    const Stage1 &s = J.st[st];
    const int Pw = st + 1 == J.nst ? P : L;
    switch (s.R) {
      case 8: stage1<T, 8, false>(s, src, dst, n, L, dL, Pw, nullptr, nullptr, nullptr, 0.0, 0.0, 0); break;
      case 4: stage1<T, 4, false>(s, src, dst, n, L, dL, Pw, nullptr, nullptr, nullptr, 0.0, 0.0, 0); break;
      case 2: stage1<T, 2, false>(s, src, dst, n, L, dL, Pw, nullptr, nullptr, nullptr, 0.0, 0.0, 0); break;
      case 3: stage1<T, 3, false>(s, src, dst, n, L, dL, Pw, nullptr, nullptr, nullptr, 0.0, 0.0, 0); break;
      case 5: stage1<T, 5, false>(s, src, dst, n, L, dL, Pw, nullptr, nullptr, nullptr, 0.0, 0.0, 0); break;
      default: stage1_generic<T>(s, src, dst, n, L, dL, Pw); break;
    }
    __syncthreads();
  }
  return dst;
}

// The tile's bootstraps b0 .. b0 + 2 np - 1 (the last one may not exist) at every point.
template <int T, bool FUSED>
__device__ __forceinline__ void vmr_points(int n, int np, int zt, int wt, int P, int b0, int nboot, double ns,
                                           double inv_ns, const double *recip, double2 *state) {
  for (int x = threadIdx.x; x < n; x += T) {
    double2 st = state[x];
    const double2 *z = sm1 + zt + x * P, *w = sm1 + wt + x * P;
    for (int q = 0; q < np; ++q) {
      const double2 zv = z[2 * q], wv = w[2 * q];
      const int b = b0 + 2 * q;
      vmr_update2<FUSED>(zv, wv, ns, inv_ns, (double)(b + 1), recip[2 * q], recip[2 * q + 1], b + 1 < nboot, st);
    }
    state[x] = st;
  }
}

// Power-of-two lines of 1024 or 2048 points: the z and the w line of a pair side by side in
// register tiles (one radix-8 butterfly a thread, n / 4 threads); the two threads that
// hold the same points of z and w exchange half of them, so each has both transforms of
// four points.  One pair at a time is all that fits with two CTAs an SM, and half of the
// general kernel's threads would idle in its radix-8 stages.  Bound by the latency of
// its shared-memory exchanges and dependent FP64 operations (40 % of the issue slots at 16 warps
// an SM).  1,024 points, 250 steps, 100 bootstraps: 0.30 ms with z and w one after the other in
// half the threads, 0.42 ms in the general kernel, 0.27 ms here, 0.23 since a NaN mean skips the IEEE
// division.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 4, LOGN == 10 ? 2 : 1)
    steps1d_pow2_kernel(const Job1 *jobs, const double2 *__restrict__ tw_g) {
  using P = Pow2<LOGN, 2>;
  using I = TileIdx<LOGN, false, 2>;
  double2 *tile = sm1, *swap = sm1 + P::TILE, *sm_tw = swap + P::N;
  const Job1 &J = jobs[blockIdx.y];
  const int s = blockIdx.x;
  if (s >= J.S) return;
  for (int i = threadIdx.x; i < P::TWSIZE; i += P::THREADS) sm_tw[i] = tw_g[i];
  const double *fz = J.fz + s * J.tab_stride, *fw = J.fw + s * J.tab_stride;
  const double cz = J.invG, cw = J.invG * J.cw[s], inv_ns = J.inv_ns;
  const int h = I::line(), t = I::bfly(), nboot = J.nboot, npairs = J.npairs;
  const double *f = h ? fw : fz;
  const double c = h ? cw : cz;
  double sc[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) sc[r] = c * __ldg(f + in_pos<LOGN>(t, r));
  double mean[4], m2[4];  // points out_pos(t, i + 4 h)
#pragma unroll
  for (int i = 0; i < 4; ++i) mean[i] = m2[i] = 0.0;
  const double2 *src = J.spectra + h * P::N;
  double2 nx[8];  // the next pair's inputs, loaded while this pair's VMR is computed
#pragma unroll
  for (int r = 0; r < 8; ++r) nx[r] = __ldg(src + in_pos<LOGN>(t, r));
  __syncthreads();
  for (int p = 0; p < npairs; ++p) {
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = cscale(nx[r], sc[r]);
    tile_fft_reg<LOGN, 1, false, 2>(tile, v, sm_tw);
    // z gives its points 4..7 for w's points 0..3
#pragma unroll
    for (int i = 0; i < 4; ++i) swap[(h * 4 + i) * P::NB8 + t] = h ? v[i] : v[i + 4];
    if (p + 1 < npairs) {
#pragma unroll
      for (int r = 0; r < 8; ++r) nx[r] = __ldg(src + (int64_t)(2 * p + 2) * P::N + in_pos<LOGN>(t, r));
    }
    __syncthreads();
    const int b = 2 * p;
    const double inv_a = 1.0 / (double)(b + 1), inv_b = 1.0 / (double)(b + 2);
    const bool has_b = b + 1 < nboot;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double2 o = swap[((1 - h) * 4 + i) * P::NB8 + t];
      const double2 z = h ? o : v[i], w = h ? v[i + 4] : o;
      double2 st = make_double2(mean[i], m2[i]);
      vmr_update2<true>(z, w, 0.0, inv_ns, 0.0, inv_a, inv_b, has_b, st);
      mean[i] = st.x;
      m2[i] = st.y;
    }
    __syncthreads();
  }
  // means: both halves transform the same line, each keeps its points
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int k = in_pos<LOGN>(t, r);
    v[r] = cscale(__ldg(J.spectra + (int64_t)(2 * npairs) * P::N + k), cz * __ldg(fz + k));
  }
  tile_fft_reg<LOGN, 1, false, 2>(tile, v, sm_tw);
  const double vs = J.vscale[s], bm1 = (double)(nboot - 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int x = h ? out_pos<LOGN>(t, i + 4) : out_pos<LOGN>(t, i);
    const double2 z = h ? v[i + 4] : v[i];
    const double var = __ddiv_rn(__dmul_rn(vs, m2[i]), bm1);
    J.f_out[(int64_t)s * P::N + x] = isfinite(var) ? log(var) : nan("");
    J.mu_out[(int64_t)s * P::N + x] = sqrt(__fma_rn(z.x, z.x, __dmul_rn(z.y, z.y)));
  }
}

// Power-of-two lines of which z and w do not fit side by side (4096 points: 74 KB each beside 65 KB of
// twiddles): z, then w in register tiles of n / 8 threads, both transforms of a thread's eight points in
// registers.  4096 points, 250 steps, 100 bootstraps, whole calls: 2.09 ms in the general kernel, whose running
// variance is in memory there, 1.20 here.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, 1)
    steps1d_line_kernel(const Job1 *jobs, const double2 *__restrict__ tw_g) {
  using P = Pow2<LOGN, 1>;
  double2 *tile = sm1, *sm_tw = sm1 + P::TILE;
  const Job1 &J = jobs[blockIdx.y];
  const int s = blockIdx.x, t = threadIdx.x;
  if (s >= J.S) return;
  for (int i = t; i < P::TWSIZE; i += P::THREADS) sm_tw[i] = tw_g[i];
  const double *fz = J.fz + s * J.tab_stride, *fw = J.fw + s * J.tab_stride;
  const double cz = J.invG, cw = J.invG * J.cw[s], inv_ns = J.inv_ns;
  const int nboot = J.nboot, npairs = J.npairs;
  double2 st[8];  // points out_pos(t, i)
#pragma unroll
  for (int i = 0; i < 8; ++i) st[i] = make_double2(0.0, 0.0);
  auto transform = [&](int64_t line, const double *f, double c, double2(&v)[8]) {
    const double2 *in = J.spectra + line * P::N;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int k = in_pos<LOGN>(t, r);
      v[r] = cscale(__ldg(in + k), c * __ldg(f + k));
    }
    tile_fft_reg<LOGN, 1, false, 1>(tile, v, sm_tw);
  };
  __syncthreads();
  for (int p = 0; p < npairs; ++p) {
    double2 z[8], w[8];
    transform(2 * p, fz, cz, z);
    transform(2 * p + 1, fw, cw, w);
    const int b = 2 * p;
    const double inv_a = 1.0 / (double)(b + 1), inv_b = 1.0 / (double)(b + 2);
    const bool has_b = b + 1 < nboot;
#pragma unroll
    for (int i = 0; i < 8; ++i) vmr_update2<true>(z[i], w[i], 0.0, inv_ns, 0.0, inv_a, inv_b, has_b, st[i]);
  }
  double2 v[8];
  transform(2 * npairs, fz, cz, v);
  const double vs = J.vscale[s], bm1 = (double)(nboot - 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int x = out_pos<LOGN>(t, i);
    const double var = __ddiv_rn(__dmul_rn(vs, st[i].y), bm1);
    J.f_out[(int64_t)s * P::N + x] = isfinite(var) ? log(var) : nan("");
    J.mu_out[(int64_t)s * P::N + x] = sqrt(__fma_rn(v[i].x, v[i].x, __dmul_rn(v[i].y, v[i].y)));
  }
}

constexpr int kPairs = 64;  // pairs per tile at most

// Any length.  Bound by instruction issue (about a third FP64) and the barriers between the
// stages; two tiles instead of one that is rewritten in place keep a thread's registers at one
// butterfly, so 32 warps share an SM (in place, with 128 registers: 16 warps, 1.4x the time).
// 250 steps, 100 bootstraps, against one launch per step and pass of a single CTA each (the
// plain form, which has the same bits): 3460 points (4 x 5 x 173) 2947 -> 22 ms.  Lengths without other
// prime factors than 2, 3 and 5 have pkde_steps1d_len.cuh.
// Shared memory: tiles a and b of n P units each; with SEQ a third one; the running
// (mean, m2) of every point where it fits (J.state null), else in global memory.
// SEQ: the z and the w line of a pair one after the other (lines too long for both).
template <int T, bool SEQ>
__global__ void __launch_bounds__(T, 1024 / T) steps1d_kernel(const Job1 *jobs) {
  __shared__ Job1 J;
  __shared__ double recip[2 * kPairs];  // 1 / i of the tile's bootstraps
  {
    const int *src = reinterpret_cast<const int *>(jobs + blockIdx.y);
    int *dst = reinterpret_cast<int *>(&J);
    for (int i = threadIdx.x; i < (int)(sizeof(Job1) / sizeof(int)); i += T) dst[i] = __ldg(src + i);
  }
  __syncthreads();
  const int s = blockIdx.x;
  if (s >= J.S) return;
  const int n = J.n, P = J.P;
  const double *fz = J.fz + s * J.tab_stride, *fw = J.fw + s * J.tab_stride;
  const double cz = J.invG, cw = J.invG * J.cw[s];
  const int ta = 0, tb = n * P, tc = 2 * n * P;
  double2 *state = SEQ ? J.state + (int64_t)s * n : sm1 + tc;
  for (int x = threadIdx.x; x < n; x += T) state[x] = make_double2(0.0, 0.0);
  for (int p0 = 0; p0 < J.npairs; p0 += J.a) {
    const int np = min(J.a, J.npairs - p0), kind = np == J.a ? 0 : 1, L = J.L[kind];
    const double2 *in = J.spectra + (int64_t)(2 * p0) * n;
    for (int l = threadIdx.x; l < 2 * np; l += T) recip[l] = 1.0 / (double)(2 * p0 + l + 1);
    int zt, wt, Pt;
    if constexpr (SEQ) {
      zt = transform1<T>(J, ta, tb, in, 1, J.dL[2], 1, fz, fz, cz, cz);
      wt = transform1<T>(J, zt == ta ? tb : ta, tc, in + n, 1, J.dL[2], 1, fw, fw, cw, cw);
      Pt = 1;
    } else {
      Pt = L == J.L[0] ? P : L | 1;
      zt = transform1<T>(J, ta, tb, in, L, J.dL[kind], Pt, fz, fw, cz, cw);
      wt = zt + 1;
    }
    if (J.fused) vmr_points<T, true>(n, np, zt, wt, Pt, 2 * p0, J.nboot, J.ns, J.inv_ns, recip, state);
    else vmr_points<T, false>(n, np, zt, wt, Pt, 2 * p0, J.nboot, J.ns, J.inv_ns, recip, state);
    __syncthreads();
  }
  const int mt = transform1<T>(J, ta, tb, J.spectra + (int64_t)(2 * J.npairs) * n, 1, J.dL[2], 1, fz, fz, cz, cz);
  const double vs = J.vscale[s], bm1 = (double)(J.nboot - 1);
  for (int x = threadIdx.x; x < n; x += T) {
    const double2 z = sm1[mt + x];
    const double v = __ddiv_rn(__dmul_rn(vs, state[x].y), bm1);
    const double yy = __dmul_rn(z.y, z.y);
    J.f_out[(int64_t)s * n + x] = isfinite(v) ? log(v) : nan("");
    J.mu_out[(int64_t)s * n + x] = sqrt(J.fused ? __fma_rn(z.x, z.x, yy) : __dadd_rn(__dmul_rn(z.x, z.x), yy));
  }
}

// Threads of a step's CTA and pairs per tile.  Two CTAs of 512 threads share an SM where
// tiles of about 4096 points fit twice, longer lines take one of 1024.  Results are read
// along the points: an odd pitch avoids bank conflicts where L >= 4.
struct Shape1 {
  int T, a, P;
  bool seq;
  size_t smem;
};
Shape1 shape1(int n, int npairs) {
  constexpr size_t two = 111 * 1024, one = 224 * 1024;  // beside the static shared memory
  auto bytes = [n](int a) { return sizeof(double2) * (size_t)n * (2 * (a > 1 ? 2 * a + 1 : 2) + 1); };
  Shape1 r{512, 1, 2, false, 0};
  if (bytes(1) <= two) {
    int most = 1;
    while (most < std::min(npairs, kPairs) && 2 * (most + 1) * n <= 4096 && bytes(most + 1) <= two) ++most;
    const int tiles = (npairs + most - 1) / most;
    r.a = (npairs + tiles - 1) / tiles;
  } else {
    r.T = 1024;
    r.seq = bytes(1) > one;
  }
  r.P = r.seq ? 1 : (r.a > 1 ? 2 * r.a + 1 : 2);
  r.smem = r.seq ? sizeof(double2) * (size_t)n * 3 : bytes(r.a);
  return r;
}

// d1 and d2 of find_stability are functions of three consecutive f alone, so the logarithms
// of a block's points are computed for kConvSteps steps by all threads, then one thread per
// point walks the steps: the walk alone is a serial chain of S steps, the logarithms were
// most of it (1,024 points, 251 steps: 0.234 -> 0.035 ms).
// Several estimations a launch: 24 of 256 to 16,384 points take 0.38 ms less than with one each.
constexpr int kConvPts = 16, kConvThreads = 256, kConvSteps = 64;
constexpr int kConvJobs = 24;  // of 136 bytes: within the 4 KB of parameters
struct ConvergeJobs {
  ConvergeJob job[kConvJobs];
  unsigned block0[kConvJobs + 1];  // blocks [block0[k], block0[k + 1]) are job k's
};
__global__ void __launch_bounds__(kConvThreads) converge_steps_kernel(const __grid_constant__ ConvergeJobs jobs) {
  __shared__ double s1[kConvSteps][kConvPts], s2[kConvSteps][kConvPts];
  int k = 0;
  while (blockIdx.x >= jobs.block0[k + 1]) ++k;
  const ConvergeJob &J = jobs.job[k];
  const int64_t G = J.G, steps_low = J.steps_low, steps_over = J.steps_over;
  const int S = J.S;
  const double *__restrict__ f_all = J.f, *__restrict__ mu_all = J.mu, *__restrict__ dlogt = J.dlogt;
  const double eps = J.eps;
  const int64_t i0 = (int64_t)(blockIdx.x - jobs.block0[k]) * kConvPts;
  const int px = threadIdx.x % kConvPts;
  const int64_t i = i0 + px;
  const bool in = i < G;
  double minimum = nan("");
  uint16_t c_low = 0, c_over = 0;
  uint8_t flag = 0;
  int32_t selected = -1;
  for (int c0 = 0; c0 < S; c0 += kConvSteps) {
    const int cn = min(kConvSteps, S - c0);
    for (int q = threadIdx.x / kConvPts; q < cn; q += kConvThreads / kConvPts) {
      const int s = c0 + q;
      double d1 = 0.0, d2 = 0.0;
      if (in) {
        const double f = f_all[(int64_t)s * G + i];
        const double f1 = s >= 1 ? f_all[(int64_t)(s - 1) * G + i] : nan("");
        const double f2 = s >= 2 ? f_all[(int64_t)(s - 2) * G + i] : nan("");
        log_differences(f, f1, f2, dlogt[s], d1, d2);
      }
      s1[q][px] = d1;
      s2[q][px] = d2;
    }
    __syncthreads();
    if (threadIdx.x < kConvPts && in) {
      for (int q = 0; q < cn; ++q) {
        const StabilityResult r =
            decide_stability(s1[q][px], s2[q][px], eps, steps_low, steps_over, minimum, c_low, c_over, flag);
        c_low = r.c_low;
        c_over = r.c_over;
        flag = r.flag;
        minimum = r.new_min;
        if (r.more_stable) selected = c0 + q;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < kConvPts && in) {
    const double last = mu_all[(int64_t)(S - 1) * G + i];
    double density = selected < 0 ? last : mu_all[(int64_t)selected * G + i];
    if (isnan(density)) density = last;  // replace_nans! (GradeProEstimator.jl:1053-1072)
    J.cs.density[i] = density;
    J.cs.selected[i] = selected < 0 ? S : selected;
  }
}

}  // namespace

// Twiddles of a radix-2/3/4/5/8 stage, [k][r - 1].
static const double2 *stage1_twiddles(pkde_ctx *ctx, int n, int R, int Ns, cudaStream_t st) {
  const std::array<int, 3> k3{n, R, Ns};
  auto it = ctx->stage_tw.find(k3);
  if (it != ctx->stage_tw.end()) return it->second.as<double2>();
  const std::vector<double2> w = make_twiddles(n);
  std::vector<double2> tw;
  const int tstep = n / (Ns * R);
  for (int k = 0; k < Ns; ++k)
    for (int r = 1; r < R; ++r) tw.push_back(w[(size_t)r * k * tstep]);
  return upload_table(ctx->stage_tw, k3, tw, st);
}

bool stages_ok(int n) { return make_plan(n).nstages <= kStages1; }

int make_stages(pkde_ctx *ctx, int n, Stage1 *stages, cudaStream_t st) {
  const FftPlan p = make_plan(n);
  int ns = 1;
  for (int q = 0; q < p.nstages; ++q) {
    const int R = p.radix[q];
    stages[q] = Stage1{R, n / R, ns, n / (ns * R), p.div_ns[q],
                       R <= 5 || R == 8 ? stage1_twiddles(ctx, n, R, ns, st) : twiddles_device(ctx, n, st)};
    ns *= R;
  }
  return p.nstages;
}

bool steps1d_ok(const pkde_grid *g) {
  return g->ndim == 1 && g->dims[0] <= 4096 && stages_ok((int)g->dims[0]);
}

const double2 *stage_twiddles_device(pkde_ctx *ctx, int logn, cudaStream_t st);

size_t steps1d_job_bytes() { return sizeof(Job1); }

void steps1d_describe(pkde_ctx *ctx, const Steps1dArgs *args, int count, void *host_jobs, Steps1dPlan &plan,
                      cudaStream_t st) {
  plan = Steps1dPlan{};
  Job1 *hj = reinterpret_cast<Job1 *>(host_jobs);
  // classes: the general kernel's three forms, the power-of-two lengths 1024, 2048 and 4096, the
  // lengths with a kernel of their own.  Register tiles of 256 points lose to the general kernel where the
  // steps do not fill the SMs (100 bootstraps, 50 steps: 0.092 ms and 0.072; 250: 0.095 and 0.101).  Of 512
  // they take less time (250: 0.119 and 0.176), but the density's last bit is another one.
  constexpr int NC = 7;
  auto class_of = [](int n, const Shape1 &sh) {
    if (steps1d_len_known(n)) return 6;
    if (n == 1024 || n == 2048 || n == 4096) return n == 1024 ? 3 : n == 2048 ? 4 : 5;
    return sh.seq ? 2 : (sh.T == 512 ? 0 : 1);
  };
  static_assert(NC == Steps1dPlan::kClasses, "classes");
  int(&first)[NC + 1] = plan.first, (&S)[NC] = plan.S;
  size_t(&smem)[NC] = plan.smem;
  int k = 0;
  std::vector<int> order(count);
  for (int e = 0; e < count; ++e) order[e] = e;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return args[x].n1 < args[y].n1; });
  for (int c = 0; c < NC; ++c) {  // the jobs of one kernel lie together
    for (int e : order) {
      const Steps1dArgs &A = args[e];
      const Shape1 sh = shape1(A.n1, A.npairs);
      if (class_of(A.n1, sh) != c) continue;
      S[c] = std::max(S[c], A.S);
      smem[c] = std::max(smem[c], sh.smem);
      Job1 J{};
      J.n = A.n1;
      J.npairs = A.npairs;
      J.nboot = A.nboot;
      J.S = A.S;
      J.a = sh.a;
      J.P = sh.P;
      J.state = A.state;
      J.fused = A.fused;
      const int rem = A.npairs % sh.a ? A.npairs % sh.a : sh.a;
      const int Ls[3] = {2 * sh.a, 2 * rem, 1};
      for (int q = 0; q < 3; ++q) {
        J.L[q] = Ls[q];
        J.dL[q] = make_fastdiv((uint32_t)Ls[q]);
      }
      J.tab_stride = A.tab_stride;
      J.spectra = A.spectra;
      J.fz = A.fz;
      J.fw = A.fw;
      J.cw = A.cw;
      J.vscale = A.vscale;
      J.invG = 1.0 / (double)A.n1;
      J.ns = (double)A.n;
      J.inv_ns = 1.0 / (double)A.n;
      J.f_out = A.f_out;
      J.mu_out = A.mu_out;
      J.nst = make_stages(ctx, A.n1, J.st, st);
      if (c == NC - 1) {
        if (plan.len.empty() || plan.len.back().n != A.n1) plan.len.push_back({A.n1, k, 0, 0});
        auto &g = plan.len.back();
        ++g.count;
        g.S = std::max(g.S, A.S);
      }
      hj[k++] = J;
    }
    first[c + 1] = k;
  }
}

void steps1d_run(pkde_ctx *ctx, const Steps1dPlan &plan, const void *dev_jobs, cudaStream_t st) {
  const int(&first)[Steps1dPlan::kClasses + 1] = plan.first;
  const int(&S)[Steps1dPlan::kClasses] = plan.S;
  const size_t(&smem)[Steps1dPlan::kClasses] = plan.smem;
  auto launch = [&](int c, int threads, size_t bytes, auto kern, auto... more) {
    const int m = first[c + 1] - first[c];
    if (!m) return;
    allow_dynamic_smem(ctx, kern, bytes);
    {
      Trace tr(ctx, PKDE_PHASE_STEP_VMR, st);
      kern<<<dim3((unsigned)S[c], (unsigned)m), threads, bytes, st>>>(
          static_cast<const Job1 *>(dev_jobs) + first[c], more...);
    }
    PKDE_CHECK_LAUNCH();
  };
  launch(0, 512, smem[0], steps1d_kernel<512, false>);
  launch(1, 1024, smem[1], steps1d_kernel<1024, false>);
  launch(2, 1024, smem[2], steps1d_kernel<1024, true>);
#define PKDE_P2(C, L)                                                                                          \
  launch(C, Pow2<L, 2>::THREADS, sizeof(double2) * (Pow2<L, 2>::TILE + Pow2<L, 2>::N + Pow2<L, 2>::TWSIZE),     \
         steps1d_pow2_kernel<L>, stage_twiddles_device(ctx, L, st));
  PKDE_P2(3, 10)
  PKDE_P2(4, 11)
#undef PKDE_P2
  launch(5, Pow2<12, 1>::THREADS, sizeof(double2) * (Pow2<12, 1>::TILE + Pow2<12, 1>::TWSIZE), steps1d_line_kernel<12>,
         stage_twiddles_device(ctx, 12, st));
  for (const auto &g : plan.len) {
    {
      Trace tr(ctx, PKDE_PHASE_STEP_VMR, st);
      steps1d_len_run(ctx, g.n, static_cast<const Job1 *>(dev_jobs) + g.first, g.count, g.S, st);
    }
    PKDE_CHECK_LAUNCH();
  }
}

// Device bytes of the running state kept in global memory (0: in shared memory).
size_t steps1d_state_bytes(int n1, int npairs, int64_t S) {
  if (steps1d_len_known(n1) || n1 == 4096) return 0;
  return shape1(n1, npairs).seq ? sizeof(double2) * (size_t)n1 * (size_t)S : 0;
}

void converge_steps(pkde_ctx *ctx, const std::vector<ConvergeJob> &all, cudaStream_t st) {
  for (size_t e = 0; e < all.size();) {
    ConvergeJobs J{};
    unsigned blocks = 0;
    for (int k = 0; k < kConvJobs; ++k) {  // the unused ones get no blocks
      J.block0[k] = blocks;
      if (e == all.size()) continue;
      const unsigned more = (unsigned)((all[e].G + kConvPts - 1) / kConvPts);
      if (k && blocks + more > 0x7fffffffu) continue;
      J.job[k] = all[e++];
      blocks += more;
    }
    J.block0[kConvJobs] = blocks;
    {
      Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
      converge_steps_kernel<<<blocks, kConvThreads, 0, st>>>(J);
    }
    PKDE_CHECK_LAUNCH();
  }
}

}  // namespace pkde
