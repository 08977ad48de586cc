// 1-D bandwidth steps of lengths known at compile time (every 2^a 3^b 5^c from 18 to 4096 that is
// not a power of two): steps1d_kernel's operations in the same order.  That kernel spends 342
// instructions a point of which 98 are FP64.  Bound by instruction issue, the latency of the stages
// at 16 warps an SM, and 251 steps on 148 SMs.  250 steps, 100 bootstraps: 500 points 0.295 ->
// 0.215 ms, 2500 points 1.61 -> 1.20 ms.
#pragma once

#include "pkde_len.cuh"
#include "pkde_steps1d.cuh"

namespace pkde {

// A tile holds L lines of n points, the z and w lines of L / 2 pairs; two tiles, two CTAs an SM.
// PAIRED false: lines of which two tiles of z and w do not fit twice, z and w one after the other,
// the points of z in registers.  Threads: the number whose passes over the stages and the points cost
// least.
template <int n>
struct OneLen {
  static constexpr LenStages S = len_stages(n);
  static constexpr bool paired = 2 * 2 * n * 16 <= 111 * 1024, two = 2 * n * 16 <= 111 * 1024;
  __host__ __device__ static constexpr int lines() {
    if (!paired) return 1;
    int L = 2;
    while (L < 128 && (L + 2) * n <= 4096 && 2 * (L + 3) * n * 16 <= 111 * 1024) L += 2;
    return L;
  }
  static constexpr int L = lines(), P = L > 2 ? L | 1 : L;
  __host__ __device__ static constexpr int threads() {
    int best = 0, best_cost = 1 << 30;
    for (int T = 256; T <= (two ? 512 : 768); T += 32) {
      int cost = 0;
      for (int i = 0; i < S.nst; ++i) cost += (n / S.rad[i] * L + T - 1) / T * (8 * S.rad[i] + 20);
      cost *= paired ? 1 : 2;
      cost += (n + T - 1) / T * (paired ? L / 2 : 1) * 60;
      if (cost < best_cost) best_cost = cost, best = T;
    }
    return best;
  }
  static constexpr int T = threads(), ctas = two ? 2 : 1, pts = (n + T - 1) / T;
  static constexpr size_t smem = sizeof(double2) * 2 * n * P;
};

extern __shared__ double2 smo[];

// The stages of a tile from I on, from the tile at `in` (I = 0: from the spectra) to `out` and back;
// the last one leaves its lines at pitch P.
template <int n, int I>
__device__ __forceinline__ void one_stages(const Job1 &J, unsigned in, unsigned out, const double2 *spectra, int most,
                                           const double *f0, const double *f1, double c0, double c1) {
  using X = OneLen<n>;
  constexpr int L = X::L, T = X::T, Q = X::S.rad[I], Ns = Len<n, 1>::ns(I), nb = n / Q;
  constexpr bool last = I + 1 == X::S.nst;
  constexpr unsigned PI = L * 16u, PO = (last ? X::P : L) * 16u;
  len_stage<T, n, Q, Ns, L>(
      J.st[I].tw,
      [&](int l, int j, double2(&v)[Q]) {
        if constexpr (I == 0) {
          const double2 *p = spectra + min(l, most) * n + j;
          const double *f = ((l & 1) ? f1 : f0) + j;
          const double c = (l & 1) ? c1 : c0;
#pragma unroll
          for (int r = 0; r < Q; ++r) {
            const double2 x = __ldg(p + r * nb);
            const double sc = c * __ldg(f + r * nb);
            v[r] = make_double2(__dmul_rn(x.x, sc), __dmul_rn(x.y, sc));
          }
        } else {
          const unsigned p = in + j * PI + l * 16u;
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = lds(p + r * nb * PI);
        }
      },
      [&](int l, int pos, double2(&v)[Q]) {
        const unsigned p = out + pos * PO + l * 16u;
#pragma unroll
        for (int q = 0; q < Q; ++q) sts(p + q * Ns * PO, v[q]);
      });
  __syncthreads();
  if constexpr (!last) one_stages<n, I + 1>(J, out, in, spectra, most, f0, f1, c0, c1);
}

// One CTA per step and job.  Line 2 npairs, the means', follows the pairs' in the last tile.  The running
// (mean, m2) of a point stays in registers.
template <int n>
__global__ void __launch_bounds__(OneLen<n>::T, OneLen<n>::ctas) steps1d_len_kernel(const Job1 *jobs) {
  using X = OneLen<n>;
  constexpr int T = X::T, L = X::L;
  __shared__ Job1 J;
  __shared__ double recip[X::paired ? L : 2];
  {
    const int *src = reinterpret_cast<const int *>(jobs + blockIdx.y);
    int *dst = reinterpret_cast<int *>(&J);
    for (int i = threadIdx.x; i < (int)(sizeof(Job1) / sizeof(int)); i += T) dst[i] = __ldg(src + i);
  }
  __syncthreads();
  const int s = blockIdx.x;
  if (s >= J.S) return;
  const double *fz = J.fz + s * J.tab_stride, *fw = J.fw + s * J.tab_stride;
  const double cz = J.invG, cw = J.invG * J.cw[s], ns = J.ns, inv_ns = J.inv_ns;
  const int npairs = J.npairs, nboot = J.nboot;
  const unsigned a = smem_of(smo), b = a + n * X::P * 16u, res = (X::S.nst & 1) ? a : b;
  double2 st[X::pts];
#pragma unroll
  for (int i = 0; i < X::pts; ++i) st[i] = make_double2(0.0, 0.0);
  auto points = [&](auto f) {
#pragma unroll
    for (int i = 0; i < X::pts; ++i) {
      const int x = (int)threadIdx.x + i * T;
      if ((i + 1) * T <= n || x < n) f(i, x);
    }
  };
  auto update = [&](double2 z, double2 w, int bt, double ra, double rb, double2 &s2) {
    vmr_update2<false>(z, w, ns, inv_ns, (double)(bt + 1), ra, rb, bt + 1 < nboot, s2);
  };
  unsigned mean = 0;  // the line of the means in the last tile, bytes
  for (int l0 = 0; l0 <= 2 * npairs; l0 += X::paired ? L : 2) {
    for (int l = threadIdx.x; l < (X::paired ? L : 2); l += T) recip[l] = 1.0 / (double)(l0 + l + 1);
    const double2 *in = J.spectra + (int64_t)l0 * n;
    if constexpr (X::paired) {
      one_stages<n, 0>(J, b, a, in, 2 * npairs - l0, fz, fw, cz, cw);
      const int np = min(L / 2, npairs - l0 / 2);
      points([&](int i, int x) {
        unsigned p = res + x * (X::P * 16u);
        for (int q = 0; q < np; ++q, p += 32u)
          update(lds(p), lds(p + 16u), l0 + 2 * q, recip[2 * q], recip[2 * q + 1], st[i]);
      });
      mean = 2 * np * 16u;
    } else {
      one_stages<n, 0>(J, b, a, in, 0, fz, fz, cz, cz);
      if (l0 < 2 * npairs) {
        double2 z[X::pts];
        points([&](int i, int x) { z[i] = lds(res + x * 16u); });
        __syncthreads();
        one_stages<n, 0>(J, b, a, in + n, 0, fw, fw, cw, cw);
        points([&](int i, int x) { update(z[i], lds(res + x * 16u), l0, recip[0], recip[1], st[i]); });
      }
    }
    if (l0 + (X::paired ? L : 2) <= 2 * npairs) __syncthreads();
  }
  const double vs = J.vscale[s], bm1 = (double)(nboot - 1);
  points([&](int i, int x) {
    const double2 z = lds(res + x * (X::P * 16u) + mean);
    const double v = __ddiv_rn(__dmul_rn(vs, st[i].y), bm1);
    J.f_out[(int64_t)s * n + x] = isfinite(v) ? log(v) : nan("");
    J.mu_out[(int64_t)s * n + x] = sqrt(__dadd_rn(__dmul_rn(z.x, z.x), __dmul_rn(z.y, z.y)));
  });
}

template <int n>
void one_run(pkde_ctx *ctx, const Job1 *jobs, int count, int S, cudaStream_t st) {
  allow_dynamic_smem(ctx, steps1d_len_kernel<n>, OneLen<n>::smem);
  steps1d_len_kernel<n><<<dim3((unsigned)S, (unsigned)count), OneLen<n>::T, OneLen<n>::smem, st>>>(jobs);
}

constexpr int kOneTable = 24;  // lengths of a source file (0: none)
struct OnePass {
  int n;
  void (*run)(pkde_ctx *, const Job1 *, int, int, cudaStream_t);
};
template <int n>
constexpr OnePass one_pass() {
  return {n, one_run<n>};
}

}  // namespace pkde
