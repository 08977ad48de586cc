// Passes of the chunked bandwidth steps (pkde_chunk.cu) along power-of-two axes whose tiles line
// up with the layout, on register tiles: one radix-8 butterfly a thread, stage outputs
// exchanged through a padded shared-memory tile (pkde_regfft.cuh).  The same operations in the
// same order as the general kernels, with every position a compile-time constant.
#include <algorithm>

#include "pkde_chunk.cuh"
#include "pkde_regfft.cuh"

namespace pkde {

const double2 *stage_twiddles_device(pkde_ctx *ctx, int logn, cudaStream_t st);

namespace {

constexpr int kT = 256;
template <int LOGN>
using PT = Pow2<LOGN, (kT * 8 >> LOGN)>;

extern __shared__ double2 smp[];

// The stages after the first one (whose outputs are v): DB as in run_stages.
template <int LOGN, int ST, bool COLS, int NL, bool DB>
__device__ __forceinline__ void p2_rest(double2 *line, double2 *line2, double2 *v, int t, const double2 *tw, int l) {
  using P = Pow2<LOGN, NL>;
  constexpr bool last8 = ST + 1 == P::NST8;
  double2 *buf = (DB && (ST & 1)) ? line2 : line;
  if constexpr (last8 && P::REM == 0) {
    if constexpr (DB && ST >= 1 && ((ST - 1) & 1) == 0) line_sync<LOGN, COLS, NL>(l);
    return;
  } else {
    stage8_store<LOGN, ST>(buf, v, t);
    line_sync<LOGN, COLS, NL>(l);
    if constexpr (!last8) {
      load8<LOGN>(buf, v, t);
      if constexpr (!DB) line_sync<LOGN, COLS, NL>(l);
      constexpr int NS = 1 << (3 * (ST + 1));
      const int k = t & (NS - 1);
      const double2 *tws = tw + P::tw_stage_off(ST + 1);
#pragma unroll
      for (int r = 1; r < 8; ++r) v[r] = cmul1(v[r], tws[(r - 1) * NS + k]);
      dft_r<8>(v);
      p2_rest<LOGN, ST + 1, COLS, NL, DB>(line, line2, v, t, tw, l);
    } else {
      constexpr int R = P::REM == 2 ? 4 : 2, NS = 1 << (3 * P::NST8), NBT = P::N / R;
      const double2 *tws = tw + P::TW8;
#pragma unroll
      for (int h = 0; h < 8 / R; ++h) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[h * R + r] = buf[pad8(t + h * P::NB8 + r * NBT)];
      }
#pragma unroll
      for (int h = 0; h < 8 / R; ++h) {
        const int k = (t + h * P::NB8) & (NS - 1);
#pragma unroll
        for (int r = 1; r < R; ++r) v[h * R + r] = cmul1(v[h * R + r], tws[(r - 1) * NS + k]);
        dft_r<R>(v + h * R);
      }
      if constexpr (!DB || (ST & 1) == 0) line_sync<LOGN, COLS, NL>(l);
    }
  }
}

template <int LOGN>
__device__ __forceinline__ void p2_twiddles(double2 *sm_tw, const double2 *tw_g) {
  for (int i = threadIdx.x; i < PT<LOGN>::TWSIZE; i += kT) sm_tw[i] = __ldg(tw_g + i);
}

// First pass, along the last axis: tile = NL adjacent lines of one array, its spectrum values held
// in registers for `per` steps of the chunk in turn (they are read once, and every step
// costs its factors, the stages and one store).
template <int LOGN>
__global__ void __launch_bounds__(kT, 2)
    p2_spectra_kernel(const __grid_constant__ AxisJob job, const double2 *__restrict__ tw_g, int per) {
  using P = PT<LOGN>;
  using I = TileIdx<LOGN, true, P::NL>;
  double2 *tile = smp, *tile2 = smp + P::TILE, *sm_tw = tile2 + P::TILE;
  const ChunkRun &run = job.run;
  const unsigned inner = job.ax.inner, G = run.G, tpa = job.ax.lines / P::NL;
  const unsigned parts = (run.C + per - 1) / per, u = blockIdx.x / parts, part = blockIdx.x - u * parts;
  const unsigned arr = u / tpa, line = (u - arr * tpa) * P::NL + I::line();
  const int t = I::bfly(), l = I::line(), ar = run.a0 + (int)arr;
  // the last axis: line index = inner index
  const double2 *in = job.in + (int64_t)ar * G + line;
  double2 raw[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) raw[r] = __ldg(in + (int64_t)in_pos<LOGN>(t, r) * inner);
  p2_twiddles<LOGN>(sm_tw, tw_g);
  unsigned at[3], li = line;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const unsigned d = q < run.N - 1 ? run.dims[q] : 1, up = li / d;
    at[q] = run.aoff[q] + (li - up * d);
    li = up;
  }
  const bool second = ar != run.mean && (ar & 1);
  const double *tab0 = second ? run.fw : run.fz;
  __syncthreads();
  const int c1 = min((int)((part + 1) * per), run.C);
  double2 *out = job.out + (int64_t)arr * G + line;
  for (int c = part * per; c < c1; ++c) {
    const int64_t s = run.s0 + c;
    const double *tab = tab0 + s * run.tab_stride;
    double f = second ? run.invG * run.cw[s] : run.invG;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (q < run.N - 1) f *= __ldg(tab + at[q]);
    const double *fl = tab + run.aoff[run.N - 1];
    double sc[8];
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      sc[r] = __ldg(fl + in_pos<LOGN>(t, r)) * f;
      v[r] = raw[r];
    }
    dft8_scaled(v, sc);
    p2_rest<LOGN, 0, true, P::NL, true>(tile + l * P::LP, tile2 + l * P::LP, v, t, sm_tw, l);
    double2 *o = out + (int64_t)c * run.A * G;
#pragma unroll
    for (int i = 0; i < 8; ++i) __stcg(o + (int64_t)out_pos<LOGN>(t, i) * inner, v[i]);
  }
}

// A later pass along an axis >= 2, in place: `per` tiles of NL adjacent lines in turn, the next
// tile's values loaded while this one is transformed.
template <int LOGN>
__global__ void __launch_bounds__(kT, 2)
    p2_axis_kernel(const __grid_constant__ AxisJob job, const double2 *__restrict__ tw_g, int per, unsigned tiles) {
  using P = PT<LOGN>;
  using I = TileIdx<LOGN, true, P::NL>;
  double2 *tile = smp, *tile2 = smp + P::TILE, *sm_tw = tile2 + P::TILE;
  const unsigned inner = job.ax.inner, G = job.run.G, tpa = job.ax.lines / P::NL;
  const int t = I::bfly(), l = I::line();
  const unsigned u0 = blockIdx.x * per, u1 = min(u0 + per, tiles);
  auto base_of = [&](unsigned u) {
    const unsigned arr = u / tpa, line = (u - arr * tpa) * P::NL + l, o = line / inner;
    return (int64_t)arr * G + (int64_t)o * P::N * inner + (line - o * inner);
  };
  int64_t base = base_of(u0);
  double2 nx[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) nx[r] = __ldcg(job.in + base + (int64_t)in_pos<LOGN>(t, r) * inner);
  p2_twiddles<LOGN>(sm_tw, tw_g);
  __syncthreads();
  for (unsigned u = u0; u < u1; ++u) {
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = nx[r];
    double2 *o = job.out + base;
    if (u + 1 < u1) {
      base = base_of(u + 1);
#pragma unroll
      for (int r = 0; r < 8; ++r) nx[r] = __ldcg(job.in + base + (int64_t)in_pos<LOGN>(t, r) * inner);
    }
    dft_r<8>(v);
    p2_rest<LOGN, 0, true, P::NL, true>(tile + l * P::LP, tile2 + l * P::LP, v, t, sm_tw, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) __stcg(o + (int64_t)out_pos<LOGN>(t, i) * inner, v[i]);
  }
}

// The z and the w line of a row: their 2 N / 8 threads meet.
template <int LOGN>
__device__ __forceinline__ void row_sync(int row) {
  constexpr int TH = (1 << LOGN) / 4;
  if constexpr (TH <= 32) __syncwarp();
  else if constexpr (TH == kT) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(9 + row), "r"(TH) : "memory");
}

// The last pass, along axis 1, of one step: rows side by side, line 2 row of a tile the z row,
// line 2 row + 1 the w row; the pairs in turn.  The two threads that hold the same points of z and w
// exchange half of them, so each has both transforms of four points and their running variance
// in registers.  The next pair's values are loaded while this one is transformed; tiles
// alternate, so one meeting per pair protects the exchange.
template <int LOGN>
__global__ void __launch_bounds__(kT, 2)
    p2_rows_kernel(const __grid_constant__ RowsJob job, const double2 *__restrict__ tw_g) {
  using P = PT<LOGN>;
  using I = TileIdx<LOGN, false, P::NL>;
  double2 *tiles = smp, *sm_tw = smp + 2 * P::TILE;
  const int G = job.G, nboot = job.nboot, per_step = job.ax.lines / (P::NL / 2);
  const unsigned c = blockIdx.x / per_step, tile = blockIdx.x - c * per_step;
  const int l = I::line(), t = I::bfly(), h = l & 1, row = l >> 1;
  const int64_t r0 = ((int64_t)tile * (P::NL / 2) + row) * P::N;
  const double2 *src = job.in + ((int64_t)c * job.A + job.arr0 + h) * G + r0;
  double2 nx[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) nx[r] = __ldcg(src + in_pos<LOGN>(t, r));
  p2_twiddles<LOGN>(sm_tw, tw_g);
  int x[4];  // this thread's points
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = h ? out_pos<LOGN>(t, i + 4) : out_pos<LOGN>(t, i);
  const int64_t o0 = (int64_t)c * G + r0;
  double2 st[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) st[i] = job.b0 > 0 ? job.state[o0 + x[i]] : make_double2(0.0, 0.0);
  __syncthreads();
  for (int p = 0; p < job.pairs; ++p) {
    double2 *mine = tiles + (p & 1) * P::TILE + l * P::LP;
    const double2 *other = tiles + (p & 1) * P::TILE + (l ^ 1) * P::LP;
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = nx[r];
    src += 2 * (int64_t)G;
    if (p + 1 < job.pairs) {
#pragma unroll
      for (int r = 0; r < 8; ++r) nx[r] = __ldcg(src + in_pos<LOGN>(t, r));
    }
    dft_r<8>(v);
    p2_rest<LOGN, 0, false, P::NL, false>(mine, nullptr, v, t, sm_tw, l);
    // z gives its points 4..7 for w's points 0..3
#pragma unroll
    for (int i = 0; i < 4; ++i) mine[i * P::NB8 + t] = h ? v[i] : v[i + 4];
    row_sync<LOGN>(row);
    const int b = job.b0 + 2 * p;
    const double ra = recip_of(job.recip, b + 1), rb = recip_of(job.recip, b + 2);
    const bool has_b = b + 1 < nboot;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double2 o = other[i * P::NB8 + t];
      const double2 z = h ? o : v[i], w = h ? v[i + 4] : o;
      double xa, xb;
      chunk_vmr2(z, w, job.inv_n, st[i].x, xa, xb);
      chunk_welford(xa, ra, st[i]);
      if (has_b) chunk_welford(xb, rb, st[i]);
    }
  }
  const bool done = job.b0 + 2 * job.pairs >= nboot;
  const double vs = job.vscale[c], bm1 = (double)(nboot - 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (done) {
      const double var = __ddiv_rn(__dmul_rn(vs, st[i].y), bm1);
      job.out[o0 + x[i]] = isfinite(var) ? log(var) : nan("");
    } else {
      job.state[o0 + x[i]] = st[i];
    }
  }
}

// The means' rows: `per` tiles of NL rows in turn, magnitudes out.
template <int LOGN>
__global__ void __launch_bounds__(kT, 2)
    p2_means_kernel(const __grid_constant__ RowsJob job, const double2 *__restrict__ tw_g, int per, unsigned tiles) {
  using P = PT<LOGN>;
  using I = TileIdx<LOGN, false, P::NL>;
  double2 *tile = smp, *sm_tw = smp + 2 * P::TILE;
  const unsigned tpa = job.ax.lines / P::NL;
  const int t = I::bfly(), l = I::line();
  const unsigned u0 = blockIdx.x * per, u1 = min(u0 + per, tiles);
  auto row_of = [&](unsigned u, unsigned &c) {
    c = u / tpa;
    return (int64_t)((u - c * tpa) * P::NL + l) * P::N;
  };
  unsigned c;
  int64_t row = row_of(u0, c);
  double2 nx[8];
  auto load = [&] {
    const double2 *src = job.in + ((int64_t)c * job.A + job.arr0) * job.G + row;
#pragma unroll
    for (int r = 0; r < 8; ++r) nx[r] = __ldcg(src + in_pos<LOGN>(t, r));
  };
  load();
  p2_twiddles<LOGN>(sm_tw, tw_g);
  __syncthreads();
  for (unsigned u = u0; u < u1; ++u) {
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = nx[r];
    double *o = job.out + (int64_t)c * job.G + row;
    if (u + 1 < u1) {
      row = row_of(u + 1, c);
      load();
    }
    dft_r<8>(v);
    p2_rest<LOGN, 0, false, P::NL, false>(tile + l * P::LP, nullptr, v, t, sm_tw, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[out_pos<LOGN>(t, i)] = sqrt(__fma_rn(v[i].x, v[i].x, __dmul_rn(v[i].y, v[i].y)));
  }
}

int log2_of(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

template <int LOGN>
size_t p2_smem() {
  return sizeof(double2) * (2 * (size_t)PT<LOGN>::TILE + PT<LOGN>::TWSIZE);
}

// Steps or tiles per CTA: as many as leave a few waves of CTAs, at most 8.
int per_cta(pkde_ctx *ctx, int64_t tiles, int64_t most) {
  return (int)std::max<int64_t>(1, std::min<int64_t>({8, most, tiles / (4 * 2 * (int64_t)ctx->sm_count)}));
}

}  // namespace

#define PKDE_P2_SWITCH(n, CALL)                                                                       \
  switch (log2_of(n)) {                                                                               \
    case 4: CALL(4); break;                                                                           \
    case 5: CALL(5); break;                                                                           \
    case 6: CALL(6); break;                                                                           \
    case 7: CALL(7); break;                                                                           \
    case 8: CALL(8); break;                                                                           \
    case 9: CALL(9); break;                                                                           \
    case 10: CALL(10); break;                                                                         \
    default: throw Error{PKDE_EUNSUPPORTED, "axis length not supported by the power-of-two passes"}; \
  }

void chunk_pow2_axis(pkde_ctx *ctx, const AxisJob &J, bool spectra, cudaStream_t st) {
  const int64_t arrays = (int64_t)J.run.A;
#define PKDE_CALL(L)                                                                                         \
  {                                                                                                          \
    const int64_t tpa = J.ax.lines / PT<L>::NL;                                                              \
    const double2 *tw = stage_twiddles_device(ctx, L, st);                                                   \
    Trace tr(ctx, PKDE_PHASE_STEP_FFT, st);                                                                  \
    if (spectra) {                                                                                           \
      const int per = per_cta(ctx, arrays * tpa * J.run.C, J.run.C);                                         \
      const unsigned parts = (unsigned)((J.run.C + per - 1) / per);                                          \
      allow_dynamic_smem(ctx, p2_spectra_kernel<L>, p2_smem<L>());                                           \
      p2_spectra_kernel<L><<<(unsigned)(arrays * tpa) * parts, kT, p2_smem<L>(), st>>>(J, tw, per);          \
    } else {                                                                                                 \
      const int64_t tiles = arrays * tpa * J.run.C;                                                          \
      const int per = per_cta(ctx, tiles, tiles);                                                            \
      allow_dynamic_smem(ctx, p2_axis_kernel<L>, p2_smem<L>());                                              \
      p2_axis_kernel<L><<<(unsigned)((tiles + per - 1) / per), kT, p2_smem<L>(), st>>>(J, tw, per,           \
                                                                                      (unsigned)tiles);      \
    }                                                                                                        \
  }
  PKDE_P2_SWITCH(J.ax.n, PKDE_CALL)
#undef PKDE_CALL
  PKDE_CHECK_LAUNCH();
}

void chunk_pow2_rows(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
#define PKDE_CALL(L)                                                                                              \
  {                                                                                                               \
    const unsigned blocks = (unsigned)(J.ax.lines / (PT<L>::NL / 2)) * J.C;                                       \
    allow_dynamic_smem(ctx, p2_rows_kernel<L>, p2_smem<L>());                                                     \
    Trace tr(ctx, PKDE_PHASE_STEP_VMR, st);                                                                       \
    p2_rows_kernel<L><<<blocks, kT, p2_smem<L>(), st>>>(J, stage_twiddles_device(ctx, L, st));                    \
  }
  PKDE_P2_SWITCH(J.ax.n, PKDE_CALL)
#undef PKDE_CALL
  PKDE_CHECK_LAUNCH();
}

void chunk_pow2_means(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
#define PKDE_CALL(L)                                                                                                \
  {                                                                                                                 \
    const int64_t tiles = (int64_t)(J.ax.lines / PT<L>::NL) * J.C;                                                  \
    const int per = per_cta(ctx, tiles, tiles);                                                                     \
    allow_dynamic_smem(ctx, p2_means_kernel<L>, p2_smem<L>());                                                      \
    Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);                                                                       \
    p2_means_kernel<L><<<(unsigned)((tiles + per - 1) / per), kT, p2_smem<L>(), st>>>(J, stage_twiddles_device(ctx, L, st), \
                                                                                     per, (unsigned)tiles);         \
  }
  PKDE_P2_SWITCH(J.ax.n, PKDE_CALL)
#undef PKDE_CALL
  PKDE_CHECK_LAUNCH();
}

}  // namespace pkde
