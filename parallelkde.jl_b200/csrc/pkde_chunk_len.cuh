// Passes of the chunked bandwidth steps (pkde_chunk.cu) for line lengths known at compile time:
// every 2^a 3^b 5^c from 18 to 1024 that is not a power of two.  The general kernels' operations in
// the same order, with every stride, division and loop bound a constant: on 100 points those
// spend 106 instructions a point, of which 29 are FP64.
#pragma once

#include <algorithm>

#include "pkde_chunk.cuh"
#include "pkde_len.cuh"

namespace pkde {

// Lines of a tile: about 800 points in multiples of eight lines (128 bytes of an element's
// lines side by side, eight lanes of a butterfly position in different banks), four lines from 257
// points on, two from 513 on.  Small tiles: more of them per SM wait at different barriers.
__host__ __device__ constexpr int len_lines(int n) {
  return n > 512 ? 2 : n > 256 ? 4 : 8 * ((800 + 4 * n) / (8 * n) > 0 ? (800 + 4 * n) / (8 * n) : 1);
}
__host__ __device__ constexpr int len_warps(int threads) {
  return threads > 256 ? 256 : (threads + 31) / 32 * 32;
}

// Twiddle tables of the stages ([k][r - 1]) and of the combine, by value of a kernel parameter.
struct LenTw {
  const double2 *st[10], *comb;
};

// All stages of L lines of n points through the tiles at byte addresses a and b in turn.
// first(l, n1, j, step, v): the inputs of butterfly j of sub-line (l, n1), elements n1 + R (j + r step);
// last(l, pos, step, v): elements pos + q step of line l.  P: pitch of the tiles (units).
template <int T, int n, int R, int L, int P, int I, class First, class Last>
__device__ __forceinline__ void len_stages_from(const LenTw &tw, unsigned in, unsigned out, const First &first,
                                                const Last &last) {
  using X = Len<n, R>;
  constexpr int M = X::M, Lr = L * R, Q = X::S.rad[I], Ns = X::ns(I);
  constexpr bool final_stage = I + 1 == X::S.nst && R == 1;
  len_stage<T, M, Q, Ns, Lr>(
      tw.st[I],
      [&](int l, int j, double2(&v)[Q]) {
        if constexpr (I == 0) {
          const int n1 = R > 1 ? l / L : 0;
          first(l - n1 * L, n1, j, std::integral_constant<int, M / Q>{}, v);
        } else {
          const unsigned p = in + (j * P + l) * 16u;
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = lds(p + r * (M / Q) * P * 16u);
        }
      },
      [&](int l, int pos, double2(&v)[Q]) {
        if constexpr (final_stage) {
          last(l, pos, std::integral_constant<int, Ns>{}, v);
        } else {
          const unsigned p = out + (pos * P + l) * 16u;
#pragma unroll
          for (int q = 0; q < Q; ++q) sts(p + q * Ns * P * 16u, v[q]);
        }
      });
  if constexpr (!final_stage) {
    __syncthreads();
    if constexpr (I + 1 < X::S.nst) {
      len_stages_from<T, n, R, L, P, I + 1>(tw, out, in, first, last);
    } else {  // combine
      constexpr int items = M * L, IT = (items + T - 1) / T;
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int e = (int)threadIdx.x + it * T;
        if ((it + 1) * T <= items || e < items) {
          const int k2 = e / L, l = e - k2 * L;
          double2 y[R];
          const unsigned p = out + (k2 * P + l) * 16u;
#pragma unroll
          for (int n1 = 0; n1 < R; ++n1) {
            y[n1] = lds(p + n1 * L * 16u);
            if (n1 > 0) y[n1] = combine_cmul(y[n1], __ldg(tw.comb + (n1 - 1) * M + k2));
          }
          dft_r<R>(y);
          last(l, k2, std::integral_constant<int, M>{}, y);
        }
      }
    }
  }
}

// The stages of a tile's lines but the last one (the combine where R > 1), element k of line l
// at unit k PN + l of `in`; the next tile is out, then in, in turn.
template <int n, int R>
__host__ __device__ constexpr int len_mids() {
  return len_stages(n / R).nst - (R > 1 ? 0 : 1);
}
template <int T, int n, int R, int L, int P, int PN, int I>
__device__ __forceinline__ void len_mid_from(const LenTw &tw, unsigned in, unsigned out) {
  if constexpr (I < len_mids<n, R>()) {
    using X = Len<n, R>;
    constexpr int M = X::M, Lr = L * R, Q = X::S.rad[I], Ns = X::ns(I);
    len_stage<T, M, Q, Ns, Lr>(
        tw.st[I],
        [&](int l, int j, double2(&v)[Q]) {
          const int n1 = R > 1 ? l / L : 0, line = l - n1 * L;
          const unsigned p = I == 0 ? in + ((n1 + j * R) * PN + line) * 16u : in + (j * P + l) * 16u;
          constexpr unsigned d = I == 0 ? M / Q * R * PN * 16u : M / Q * P * 16u;
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = lds(p + r * d);
        },
        [&](int l, int pos, double2(&v)[Q]) {
          const unsigned p = out + (pos * P + l) * 16u;
#pragma unroll
          for (int q = 0; q < Q; ++q) sts(p + q * Ns * P * 16u, v[q]);
        });
    __syncthreads();
    len_mid_from<T, n, R, L, P, PN, I + 1>(tw, out, in);
  }
}
// Radix and butterflies of the last stage; its butterfly j of line l from the tile: inputs of two
// lines of the same index, `gap` bytes apart (one set of twiddles), outputs j + q nb.
template <int n, int R>
struct LenLast {
  static constexpr int Q = R > 1 ? R : len_stages(n).rad[len_mids<n, R>()], nb = n / Q;
};
template <int n, int R, int L, int P>
__device__ __forceinline__ void len_last2(const LenTw &tw, unsigned tile, int l, int j, unsigned gap,
                                          double2 (&z)[LenLast<n, R>::Q], double2 (&w)[LenLast<n, R>::Q]) {
  constexpr int Q = LenLast<n, R>::Q, nb = LenLast<n, R>::nb;
  const unsigned p = tile + (j * P + l) * 16u;
  constexpr unsigned d = R > 1 ? L * 16u : nb * P * 16u;
#pragma unroll
  for (int r = 0; r < Q; ++r) {
    z[r] = lds(p + r * d);
    w[r] = lds(p + r * d + gap);
  }
  if constexpr (R > 1) {
#pragma unroll
    for (int r = 1; r < Q; ++r) {
      const double2 t = __ldg(tw.comb + (r - 1) * nb + j);
      z[r] = combine_cmul(z[r], t);
      w[r] = combine_cmul(w[r], t);
    }
  } else if (j > 0) {
#pragma unroll
    for (int r = 1; r < Q; ++r) {
      const double2 t = __ldg(tw.st[len_mids<n, R>()] + j * (Q - 1) + r - 1);
      z[r] = cmul1(z[r], t);
      w[r] = cmul1(w[r], t);
    }
  }
  dft_r<Q>(z);
  dft_r<Q>(w);
}

// Tiles a pass that reads and writes global memory goes through.
template <int n, int R>
__host__ __device__ constexpr int len_held() {
  const int exchanges = len_stages(n / R).nst + (R > 1 ? 1 : 0) - 1;
  return exchanges < 2 ? exchanges : 2;
}

extern __shared__ double2 sml[];

template <int n, int R>
struct AxisLen {
  // About six points a thread: 96^3, 32 bootstraps, 100 steps, tiles of 8 lines, both passes: 37.3 ms
  // with 96 threads, 30 with 128, 32.4 with 160.
  static constexpr int L = len_lines(n), T = len_warps(n * L * 4 / 25), ctas = 768 / T;
  static constexpr size_t smem = sizeof(double2) * len_held<n, R>() * n * L + 24 * L;
};

// Inverse FFT along one axis >= 2 (chunk_axis_kernel's job): a tile of L lines of a step's flattened
// (array, line) index, in `per` steps of the chunk in turn -- its line offsets are the same in
// each, and the spectra of the first pass come from the L1 or L2 after the first step.
template <int n, int R, bool SPECTRA>
__global__ void __launch_bounds__(AxisLen<n, R>::T, AxisLen<n, R>::ctas)
    len_axis_kernel(const __grid_constant__ AxisJob job, const __grid_constant__ LenTw tw, int per) {
  using X = AxisLen<n, R>;
  constexpr int T = X::T, L = X::L;
  const ChunkRun &run = job.run;
  const double **sf = reinterpret_cast<const double **>(sml + len_held<n, R>() * n * L);  // factors of the line's elements
  double *sc = reinterpret_cast<double *>(sf + L);                                     // and of its other axes
  unsigned *off = reinterpret_cast<unsigned *>(sc + L);  // bytes from the tile's first array
  unsigned *at = off + L;                                // line of its array | second array of a pair << 31
  const unsigned G = run.G, lines = job.ax.lines, inner = job.ax.inner;
  const unsigned parts = (run.C + per - 1) / per, tile = blockIdx.x / parts, part = blockIdx.x - tile * parts;
  const unsigned w0 = tile * L, arr0 = w0 / lines, li0 = w0 - arr0 * lines;
  const int valid = (int)min((unsigned)L, (unsigned)run.A * lines - w0);
  for (int l = threadIdx.x; l < L; l += T) {
    unsigned arr = arr0, li = li0 + (l < valid ? l : 0);
    while (li >= lines) li -= lines, ++arr;
    const unsigned o = li / inner;
    off[l] = ((arr - arr0) * G + o * (n * inner) + (li - o * inner)) * 16u;
    const int ar = run.a0 + (int)arr;
    at[l] = li | (ar != run.mean && (ar & 1) ? 1u << 31 : 0u);
  }
  const unsigned ss = inner * 16u, a = smem_of(sml), b = a + (len_held<n, R>() > 1 ? n * L * 16u : 0u);
  const int c1 = min((int)((part + 1) * per), run.C);
  for (int c = part * per; c < c1; ++c) {
    if constexpr (SPECTRA) {
      const int64_t s = run.s0 + c;
      for (int l = threadIdx.x; l < L; l += T) {  // the line's factors of this step (its own entries)
        const bool second = at[l] >> 31;
        unsigned li = at[l] & 0x7fffffffu;
        const double *tab = (second ? run.fw : run.fz) + s * run.tab_stride;
        double f = second ? run.invG * run.cw[s] : run.invG;
        for (int q = 0; q < run.N - 1; ++q) {
          const unsigned d = run.dims[q], up = li / d;
          f *= __ldg(tab + run.aoff[q] + (li - up * d));
          li = up;
        }
        sf[l] = tab + run.aoff[run.N - 1];
        sc[l] = f;
      }
    }
    __syncthreads();
    const int64_t base = (int64_t)(c * run.A + arr0) * G;
    const char *in = reinterpret_cast<const char *>(job.in + (SPECTRA ? (int64_t)(run.a0 + arr0) * G : base));
    char *out = reinterpret_cast<char *>(job.out + base);
    len_stages_from<T, n, R, L, L * R, 0>(
        tw, b, a,
        [&](int l, int n1, int j, auto step, auto &v) {
          constexpr int Q = sizeof(v) / sizeof(double2), d = decltype(step)::value * R;
          unsigned p = off[l] + (n1 + j * R) * ss;
#pragma unroll
          for (int r = 0; r < Q; ++r, p += d * ss) {
            const double2 *q = reinterpret_cast<const double2 *>(in + p);
            v[r] = SPECTRA ? __ldg(q) : __ldcg(q);
          }
          if constexpr (SPECTRA) {
            const double cl = sc[l];
            const double *f = sf[l] + n1 + j * R;
#pragma unroll
            for (int r = 0; r < Q; ++r) {
              const double s = __ldg(f + r * d) * cl;
              v[r] = make_double2(__dmul_rn(v[r].x, s), __dmul_rn(v[r].y, s));
            }
          }
        },
        [&](int l, int pos, auto step, auto &v) {
          constexpr int Q = sizeof(v) / sizeof(double2), d = decltype(step)::value;
          if (l < valid) {
            unsigned p = off[l] + pos * ss;
#pragma unroll
            for (int q = 0; q < Q; ++q, p += d * ss) __stcg(reinterpret_cast<double2 *>(out + p), v[q]);
          }
        });
    __syncthreads();
  }
}

template <int n, int R>
struct RowsLen {
  // One butterfly of radix 5 or two of radix 3 of the last stage a thread (its running variances
  // are registers): 100 x 100, 100 bootstraps, 250 steps, tiles of 8 lines: 1.53 ms with 96 threads, 2.0
  // with 64, 1.74 with 160; 96^3, 32, 100: 16.0 with 64, 16.8 with 96, 17.2 with 128.
  static constexpr int L = len_lines(n), rt = L / 2, last = n / LenLast<n, R>::Q * rt;
  static constexpr int T = len_warps(LenLast<n, R>::Q == 3 ? last / 2 : last), ctas = 640 / T;
  // lines of a tile: z row l at l zs, its w row `gap` lines on, so that eight lanes of the last stage (rows,
  // then butterflies) meet different banks: side by side for 4 rows, the z rows first else
  static constexpr int zs = rt == 4 ? 2 : 1, gap = rt == 4 ? 1 : rt;
  static constexpr int PN = L | 1, P = (L * R) | 1;
  static constexpr int size = n * PN > n / R * P ? n * PN : n / R * P;
  static constexpr size_t smem = sizeof(double2) * 2 * size;
};

// The rows [row0, + count / n) of a tile into shared memory, element k of line l at unit k PN + l;
// (row l: line l zs; with a gap the next array's rows too, gap lines on).
template <int n, int T, int most, unsigned PN, int zs, int gap>
__device__ __forceinline__ void len_load_rows(unsigned tile, const double2 *z, int count, int64_t G) {
#pragma unroll
  for (int q = 0; q < (most * n + T - 1) / T; ++q) {
    const int e = (int)threadIdx.x + q * T, l = e / n;
    if (e < count) {
      const unsigned p = tile + ((e - l * n) * PN + l * zs) * 16u;
      cp_async16(p, z + e);
      if (gap) cp_async16(p + gap * 16u, z + G + e);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// The z and w rows of a tile, pairs in turn (rows_body of pkde_chunk.cu).  A thread takes the last
// butterfly of a z row and that of its w row, so the variance-to-mean ratios and their running
// variance need no exchange: 24 shared-memory wavefronts a point against 32 (the kernels are
// bound by those and by latency, at 30 % of the issue slots), and the tile that the last
// stage does not read takes the next pair's rows meanwhile.  96^3 (above): 23 ms in the general
// kernel, 20 with the ratios after an exchange, 16 here.
template <int n, int R>
__global__ void __launch_bounds__(RowsLen<n, R>::T, RowsLen<n, R>::ctas)
    len_rows_kernel(const __grid_constant__ RowsJob job, const __grid_constant__ LenTw tw, int tiles) {
  using X = RowsLen<n, R>;
  constexpr int T = X::T, L = X::L, rt = X::rt, Q = LenLast<n, R>::Q, nb = LenLast<n, R>::nb;
  constexpr int items = nb * rt, IT = (items + T - 1) / T;
  const int G = job.G, nboot = job.nboot;
  const unsigned bz = blockIdx.x / (unsigned)tiles, bx = blockIdx.x - bz * tiles;
  const int row0 = bx * rt, rows = min(rt, job.ax.lines - row0);
  const double2 *z = job.in + ((int64_t)bz * job.A + job.arr0) * G + (int64_t)row0 * n;
  unsigned cur = smem_of(sml);
  const unsigned both = 2 * cur + X::size * 16u;
  len_load_rows<n, T, rt, X::PN, X::zs, X::gap>(cur, z, rows * n, G);
  const int64_t o0 = (int64_t)bz * G + (int64_t)row0 * n;
  double2 st[IT][Q];
  auto each = [&](auto f) {  // f(it, l, j): this thread's butterflies of the last stage
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int e = (int)threadIdx.x + it * T, j = e / rt, l = e - j * rt;
      if (((it + 1) * T <= items || e < items) && l < rows) f(it, l, j);
    }
  };
#pragma unroll
  for (int it = 0; it < IT; ++it)
#pragma unroll
    for (int q = 0; q < Q; ++q) st[it][q] = make_double2(0.0, 0.0);
  if (job.b0 > 0)
    each([&](int it, int l, int j) {
#pragma unroll
      for (int q = 0; q < Q; ++q) st[it][q] = job.state[o0 + l * n + j + q * nb];
    });
  for (int p = 0; p < job.pairs; ++p) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    len_mid_from<T, n, R, L, X::P, X::PN, 0>(tw, cur, both - cur);
    const unsigned res = (len_mids<n, R>() & 1) ? both - cur : cur;
    cur = both - res;
    z += 2 * (int64_t)G;
    if (p + 1 < job.pairs) len_load_rows<n, T, rt, X::PN, X::zs, X::gap>(cur, z, rows * n, G);
    const int b = job.b0 + 2 * p;
    const double ra = recip_of(job.recip, b + 1), rb = recip_of(job.recip, b + 2);
    const bool has_b = b + 1 < nboot;
    each([&](int it, int l, int j) {
      double2 zv[Q], wv[Q];
      len_last2<n, R, L, X::P>(tw, res, l * X::zs, j, X::gap * 16u, zv, wv);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        double xa, xb;
        chunk_vmr2(zv[q], wv[q], job.inv_n, st[it][q].x, xa, xb);
        chunk_welford(xa, ra, st[it][q]);
        if (has_b) chunk_welford(xb, rb, st[it][q]);
      }
    });
  }
  const bool done = job.b0 + 2 * job.pairs >= nboot;
  const double vs = job.vscale[bz], bm1 = (double)(nboot - 1);
  each([&](int it, int l, int j) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t o = o0 + l * n + j + q * nb;
      if (done) {
        const double v = __ddiv_rn(__dmul_rn(vs, st[it][q].y), bm1);
        job.out[o] = isfinite(v) ? log(v) : nan("");
      } else {
        job.state[o] = st[it][q];
      }
    }
  });
}

// Rows of the means' array and their magnitudes: a tile of L rows in `per` steps in turn, the next
// step's rows coming in by cp.async meanwhile.
template <int n, int R>
__global__ void __launch_bounds__(RowsLen<n, R>::T, RowsLen<n, R>::ctas)
    len_means_kernel(const __grid_constant__ RowsJob job, const __grid_constant__ LenTw tw, int tiles, int per) {
  using X = RowsLen<n, R>;
  constexpr int T = X::T, L = X::L, PTS = (L * n + T - 1) / T;
  constexpr unsigned PB = X::PN * 16u, tsize = X::size * 16u;
  const int G = job.G;
  const unsigned part = blockIdx.x / (unsigned)tiles, bx = blockIdx.x - part * tiles;
  const int row0 = bx * L, count = min(L, job.ax.lines - row0) * n;
  const int c0 = part * per, c1 = min(c0 + per, job.C);
  const double2 *z = job.in + ((int64_t)c0 * job.A + job.arr0) * G + (int64_t)row0 * n;
  double *out = job.out + (int64_t)c0 * G + (int64_t)row0 * n;
  auto at = [](int e) {
    const int l = e / n;
    return (e - l * n) * PB + l * 16u;
  };
  auto load = [&](unsigned tile) { len_load_rows<n, T, L, X::PN, 1, 0>(tile, z, count, 0); };
  constexpr int total = len_stages(n / R).nst + (R > 1 ? 1 : 0);
  unsigned cur = smem_of(sml);
  const unsigned both = 2 * cur + tsize;
  load(cur);
  for (int c = c0; c < c1; ++c) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const unsigned src = cur, res = (total & 1) ? both - cur : cur;
    len_stages_from<T, n, R, L, X::P, 0>(
        tw, src, both - src,
        [&](int l, int n1, int j, auto step, auto &v) {
          constexpr int Q = sizeof(v) / sizeof(double2), d = decltype(step)::value * R;
          const unsigned q = src + (n1 + j * R) * PB + l * 16u;
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = lds(q + r * d * PB);
        },
        [&](int l, int pos, auto step, auto &v) {
          constexpr int Q = sizeof(v) / sizeof(double2), d = decltype(step)::value;
          const unsigned o = res + pos * PB + l * 16u;
#pragma unroll
          for (int q = 0; q < Q; ++q) sts(o + q * d * PB, v[q]);
        });
    __syncthreads();
    cur = both - res;
    z += (int64_t)job.A * G;
    if (c + 1 < c1) load(cur);
#pragma unroll
    for (int q = 0; q < PTS; ++q) {
      const int e = (int)threadIdx.x + q * T;
      if (e < count) {
        const double2 v = lds(res + at(e));
        out[e] = sqrt(__fma_rn(v.x, v.x, __dmul_rn(v.y, v.y)));
      }
    }
    out += G;
  }
}

inline LenTw len_twiddles(const ChunkAxis &ax) {
  LenTw tw{};
  for (int i = 0; i < ax.nst; ++i) tw.st[i] = ax.st[i].tw;
  tw.comb = ax.twc;
  return tw;
}

// Steps per CTA of a pass: as many as leave four waves of CTAs, at most 8.
inline int len_per(pkde_ctx *ctx, int64_t tiles, int C, int ctas) {
  return (int)std::max<int64_t>(1, std::min<int64_t>({8, C, tiles * C / (4 * ctas * (int64_t)ctx->sm_count)}));
}

template <int n, int R>
void len_axis(pkde_ctx *ctx, const AxisJob &J, bool spectra, cudaStream_t st) {
  using X = AxisLen<n, R>;
  const int64_t tiles = ((int64_t)J.run.A * J.ax.lines + X::L - 1) / X::L;
  const int per = len_per(ctx, tiles, J.run.C, X::ctas);
  const unsigned blocks = (unsigned)(tiles * ((J.run.C + per - 1) / per));
  auto kern = spectra ? len_axis_kernel<n, R, true> : len_axis_kernel<n, R, false>;
  allow_dynamic_smem(ctx, kern, X::smem);
  Trace tr(ctx, PKDE_PHASE_STEP_FFT, st);
  kern<<<blocks, X::T, X::smem, st>>>(J, len_twiddles(J.ax), per);
}

template <int n, int R>
void len_rows(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
  using X = RowsLen<n, R>;
  const int tiles = (J.ax.lines + X::rt - 1) / X::rt;
  allow_dynamic_smem(ctx, len_rows_kernel<n, R>, X::smem);
  Trace tr(ctx, PKDE_PHASE_STEP_VMR, st);
  len_rows_kernel<n, R><<<(unsigned)(tiles * J.C), X::T, X::smem, st>>>(J, len_twiddles(J.ax), tiles);
}

template <int n, int R>
void len_means(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
  using X = RowsLen<n, R>;
  const int tiles = (J.ax.lines + X::L - 1) / X::L, per = len_per(ctx, tiles, J.C, X::ctas);
  const unsigned blocks = (unsigned)(tiles * ((J.C + per - 1) / per));
  allow_dynamic_smem(ctx, len_means_kernel<n, R>, X::smem);
  Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
  len_means_kernel<n, R><<<blocks, X::T, X::smem, st>>>(J, len_twiddles(J.ax), tiles, per);
}

// 3 2^m and 5 2^m from 2^3 on: interleaved sub-lines (mix_radix of the engine); else one line.
__host__ __device__ constexpr int len_radix(int n) {
  for (int r = 3; r <= 5; r += 2)
    if (n % r == 0 && n / r >= 8 && (n / r & (n / r - 1)) == 0) return r;
  return 1;
}

constexpr int kLenTable = 18;  // lengths of a source file (0: none)

// The launchers of one length.
struct LenPasses {
  int n, R;
  void (*axis)(pkde_ctx *, const AxisJob &, bool, cudaStream_t);
  void (*rows)(pkde_ctx *, const RowsJob &, cudaStream_t);
  void (*means)(pkde_ctx *, const RowsJob &, cudaStream_t);
};
template <int n>
constexpr LenPasses len_passes() {
  constexpr int R = len_radix(n);
  return {n, R, len_axis<n, R>, len_rows<n, R>, len_means<n, R>};
}

}  // namespace pkde
