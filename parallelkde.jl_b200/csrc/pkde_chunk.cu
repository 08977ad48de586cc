// Bandwidth steps of N-D estimations (N >= 2) several steps at a time: one launch per pass
// for a chunk of steps and bootstrap pairs whose intermediates stay in the L2.
//
//   chunk_axis_kernel   inverse FFT along axes N..2, the propagation factors applied on
//                       the first load (FourierSpace.jl:215-262, :445-524);
//   chunk_rows_kernel   inverse FFT along axis 1 of the z and w rows of a few pairs, the
//                       variance-to-mean ratio of each bootstrap (DirectSpace.jl:550-552),
//                       or of the means' rows (:747-764);
//   chunk_var_kernel    the running variance over the bootstraps in order and the log
//                       scaled variance of every point (:544-581);
//   then the convergence walk (:829-1031), over all steps at the end where f and the
//   means of every step fit in memory, else chunk by chunk.
//
// The steps are independent given the spectra, so a chunk has no ordering inside it: the
// launches need no dependency counters, and every axis length fills its tiles (2048
// points, as many lines as fit, lines of different arrays and steps side by side).
// The persistent engine (pkde_engine.cu) keeps the shapes whose tiles it fills itself.
#include <algorithm>

#include "pkde_lines.cuh"
#include "pkde_step.cuh"

namespace pkde {
namespace {

constexpr int kCT = 256;       // threads
constexpr int kTilePts = 2048; // points per tile

// One grid axis.  Lines of n = R M points: R = 1, plain Stockham stages; R = 3 or 5 (M a power
// of two from 8), the R interleaved sub-lines x[R n2 + n1] through the stages of M, then
// one radix-R combine X[k2 + M q] = sum_n1 W_n^(n1 k2) Y_n1[k2] W_R^(n1 q) (the step
// engine's mixed-radix arithmetic).
struct ChunkAxis {
  int n, M, R, nst, inner, lines;
  int generic_first;   // the first stage has a generic radix: one more exchange
  int fused;           // the first stage's sums fuse the scaling of one operand (power-of-two register tiles)
  const double2 *twc;  // combine twiddles [n1 - 1][k2]
  Stage1 st[kStages1];
};
// Lines of a tile: L (pitch PN where a tile holds lines), Lr = L R sub-lines (pitch P); size: units
// of one tile.
struct ChunkTile {
  int L, Lr, P, PN, size;
  FastDiv dL, dLr;
};

struct ChunkRun {
  int N, G, A, a0, C, mean;  // A arrays from a0 per step, C steps from s0; mean: index of the means' array
  int64_t s0, tab_stride;
  const double *fz, *fw, *cw;
  double invG;
  int dims[4];
  int64_t aoff[4];
};

// Tiles an axis pass holds: the first stage reads global memory and the last one writes it.
__host__ __device__ __forceinline__ int axis_tiles_held(const ChunkAxis &ax) {
  const int exchanges = ax.nst + (ax.R > 1 ? 1 : 0) - 1 + ax.generic_first;
  return exchanges < 2 ? exchanges : 2;
}

extern __shared__ double2 smc[];

// Lines through every stage: input element k of line l at src(l) + k ss (loaded by ld, scaled by
// scale(l) and f[k] where `scaled`), tiles a and b in turn, output position p of line l through
// st(l, p, value).  Every thread calls; the caller synchronises before the tiles are reused.
template <class Src, class Ld, class Fac, class St>
__device__ __forceinline__ void chunk_transform(const ChunkAxis &ax, const ChunkTile &t, double2 *a, double2 *b,
                                                int64_t ss, Src src, Ld ld, bool scaled, Fac fac, St st) {
  const int R = ax.R, L = t.L, Lr = t.Lr, P = t.P;
  const int total = ax.nst + (R > 1 ? 1 : 0);
  auto sub = [&](int l, int &n1) {  // sub-line l = n1 L + line
    n1 = R > 1 ? (int)fdiv((uint32_t)l, t.dL) : 0;
    return l - n1 * L;
  };
  int s0 = 0;
  double2 *in = b, *out = a;
  const int64_t rs = ss * R;
  if (ax.generic_first) {  // its inputs pass through the tile (R = 1)
    for (int e = threadIdx.x; e < ax.n * L; e += kCT) {
      const int k = (int)fdiv((uint32_t)e, t.dL), l = e - k * L;
      double2 v = ld(src(l) + k * ss);
      if (scaled) {
        double c;
        const double *f = fac(l, c);
        const double sc = __ldg(f + k) * c;
        v = make_double2(__dmul_rn(v.x, sc), __dmul_rn(v.y, sc));
      }
      out[k * P + l] = v;
    }
    __syncthreads();
    in = a;
    out = b;
  } else {
    const Stage1 &s = ax.st[0];
    auto first = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      auto load = [&](int j, int l, double2(&v)[Q]) {
        int n1;
        const int line = sub(l, n1);
        const double2 *p = src(line) + n1 * ss + (int64_t)j * rs;
        const int64_t step = s.nb * rs;
#pragma unroll
        for (int r = 0; r < Q; ++r) v[r] = ld(p + r * step);
        if (scaled) {
          double c;
          const double *f = fac(line, c) + n1 + j * R;
          double sc[Q];
#pragma unroll
          for (int r = 0; r < Q; ++r) sc[r] = __ldg(f + r * s.nb * R) * c;
          if constexpr (Q == 8) {
            if (ax.fused) {
              dft8_scaled(v, sc);
              return true;
            }
          }
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = make_double2(__dmul_rn(v[r].x, sc[r]), __dmul_rn(v[r].y, sc[r]));
        }
        return false;
      };
      if (total == 1) {
        line_stage<kCT, Q>(s, Lr, t.dLr, true, load, [&](int l, int pos, double2(&v)[Q]) {
#pragma unroll
          for (int q = 0; q < Q; ++q) st(l, pos + q, v[q]);
        });
      } else {
        line_stage<kCT, Q>(s, Lr, t.dLr, true, load, [&](int l, int pos, double2(&v)[Q]) {
          double2 *o = out + pos * P + l;
#pragma unroll
          for (int q = 0; q < Q; ++q) o[q * P] = v[q];
        });
      }
    };
    switch (s.R) {
      case 8: first(std::integral_constant<int, 8>{}); break;
      case 4: first(std::integral_constant<int, 4>{}); break;
      case 2: first(std::integral_constant<int, 2>{}); break;
      case 3: first(std::integral_constant<int, 3>{}); break;
      default: first(std::integral_constant<int, 5>{}); break;
    }
    if (total > 1) __syncthreads();
    in = a;
    out = b;
    s0 = 1;
  }
  for (int i = s0; i < ax.nst; ++i) {
    const Stage1 &s = ax.st[i];
    const bool last = i + 1 == total;
    auto stage = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      auto load = [&](int j, int l, double2(&v)[Q]) {
        const double2 *p = in + j * P + l;
        const int step = s.nb * P;
#pragma unroll
        for (int r = 0; r < Q; ++r) v[r] = p[r * step];
        return false;
      };
      if (last) {
        line_stage<kCT, Q>(s, Lr, t.dLr, false, load, [&](int l, int pos, double2(&v)[Q]) {
#pragma unroll
          for (int q = 0; q < Q; ++q) st(l, pos + q * s.Ns, v[q]);
        });
      } else {
        line_stage<kCT, Q>(s, Lr, t.dLr, false, load, [&](int l, int pos, double2(&v)[Q]) {
          double2 *o = out + pos * P + l;
          const int step = s.Ns * P;
#pragma unroll
          for (int q = 0; q < Q; ++q) o[q * step] = v[q];
        });
      }
    };
    switch (s.R) {
      case 8: stage(std::integral_constant<int, 8>{}); break;
      case 4: stage(std::integral_constant<int, 4>{}); break;
      case 2: stage(std::integral_constant<int, 2>{}); break;
      case 3: stage(std::integral_constant<int, 3>{}); break;
      case 5: stage(std::integral_constant<int, 5>{}); break;
      default:
        if (last) line_stage_generic<kCT>(s, ax.n, Lr, t.dLr, in, P, st);
        else line_stage_generic<kCT>(s, ax.n, Lr, t.dLr, in, P, [&](int l, int pos, double2 v) { out[pos * P + l] = v; });
        break;
    }
    if (!last) __syncthreads();
    double2 *x = in;
    in = out;
    out = x;
  }
  if (R > 1) {
    auto combine = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      const int M = ax.M, items = M * L;
      for (int e = threadIdx.x; e < items; e += kCT) {
        const int k2 = (int)fdiv((uint32_t)e, t.dL), l = e - k2 * L;
        double2 y[Q];
#pragma unroll
        for (int n1 = 0; n1 < Q; ++n1) {
          y[n1] = in[k2 * P + n1 * L + l];
          if (n1 > 0) {  // the engine's combine fuses the other product of the imaginary part
            const double2 v = y[n1], w = __ldg(ax.twc + (n1 - 1) * M + k2);
            y[n1] = make_double2(__fma_rn(v.x, w.x, -__dmul_rn(v.y, w.y)), __fma_rn(v.x, w.y, __dmul_rn(v.y, w.x)));
          }
        }
        dft_r<Q>(y);
#pragma unroll
        for (int q = 0; q < Q; ++q) st(l, k2 + M * q, y[q]);
      }
    };
    if (R == 3) combine(std::integral_constant<int, 3>{});
    else combine(std::integral_constant<int, 5>{});
  }
}

// Inverse FFT along one axis >= 2 of A arrays in each of C steps: tile = L consecutive lines
// of the flattened (step, array, line) index.  SPECTRA: the first pass, from the spectra,
// with the factors of every axis and the array's scalar; else in place.
template <bool SPECTRA>
__global__ void __launch_bounds__(kCT, 3)
    chunk_axis_kernel(const __grid_constant__ ChunkAxis ax, const __grid_constant__ ChunkTile t,
                      const __grid_constant__ ChunkRun run, const double2 *in, double2 *out) {
  double2 *a = smc, *b = a + t.size;
  int64_t *so = reinterpret_cast<int64_t *>(smc + axis_tiles_held(ax) * t.size);
  int64_t *si = so + t.L;
  const double **sf = reinterpret_cast<const double **>(si + t.L);
  double *sc = reinterpret_cast<double *>(sf + t.L);
  const int G = run.G;
  {
    const unsigned per = (unsigned)run.A * ax.lines, total = (unsigned)run.C * per;
    for (int l = threadIdx.x; l < t.L; l += kCT) {
      unsigned w = blockIdx.x * (unsigned)t.L + l;
      const bool valid = w < total;
      if (!valid) w = 0;
      const unsigned c = w / per, r = w - c * per, arr = r / ax.lines;
      unsigned li = r - arr * ax.lines;
      const int64_t off = (int64_t)(li / ax.inner) * ax.n * ax.inner + li % ax.inner;
      const int64_t dst = (int64_t)(c * run.A + arr) * G + off;
      so[l] = valid ? dst : -1;
      si[l] = SPECTRA ? (int64_t)(run.a0 + arr) * G + off : dst;
      if (SPECTRA) {
        const int64_t s = run.s0 + c;
        const int ar = run.a0 + (int)arr;
        const bool second = ar != run.mean && (ar & 1);
        const double *tab = (second ? run.fw : run.fz) + s * run.tab_stride;
        double f = second ? run.invG * run.cw[s] : run.invG;
        for (int q = 0; q < run.N - 1; ++q) {
          f *= tab[run.aoff[q] + li % run.dims[q]];
          li /= run.dims[q];
        }
        sf[l] = tab + run.aoff[run.N - 1];
        sc[l] = f;
      }
    }
  }
  __syncthreads();
  chunk_transform(
      ax, t, a, b, ax.inner, [&](int l) { return in + si[l]; },
      [](const double2 *p) { return SPECTRA ? __ldg(p) : __ldcg(p); }, SPECTRA,
      [&](int l, double &c) {
        c = sc[l];
        return sf[l];
      },
      [&](int l, int pos, double2 v) {
        const int64_t o = so[l];
        if (o >= 0) __stcg(out + o + (int64_t)pos * ax.inner, v);
      });
}

__device__ __forceinline__ double chunk_vmr(double Mv, double Vv, double inv_n) {
  const double m = __dmul_rn(fabs(Mv), inv_n);
  return div_nr(__fma_rn(-m, m, __dmul_rn(fabs(Vv), inv_n)), m);
}

__device__ __forceinline__ void cp_async16(double2 *dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Inverse FFT along axis 1.  Tile = rows [blockIdx.x rt, + rt) of step blockIdx.z.  VMR: the z
// and w rows of pairs [blockIdx.y np, + np) of the chunk's `pairs`, line l < rt the z row l,
// line rt + l its w row; x[(step B + bootstrap) G + point] = the bootstrap's VMR.  The rows
// of the next pair come in by cp.async while the VMR of this one is computed.  Else
// the rows of the means' array, mu[step G + point] = their magnitudes.
template <bool VMR>
__global__ void __launch_bounds__(kCT, 3)
    chunk_rows_kernel(const __grid_constant__ ChunkAxis ax, const __grid_constant__ ChunkTile t, int G, int A, int arr0,
                      int rt, int pairs, int np, int b0, int nboot, double inv_n, const double2 *in, double *out) {
  const int n = ax.n, PN = t.PN, row0 = blockIdx.x * rt, nrow = min(rt, ax.lines - row0);
  const int p0 = VMR ? blockIdx.y * np : 0, p1 = VMR ? min(p0 + np, pairs) : 1;
  const double2 *base = in + ((int64_t)blockIdx.z * A + arr0) * G + (int64_t)row0 * n;
  double2 *buf[2] = {smc, smc + t.size};
  auto load = [&](int p, double2 *dst) {
    const double2 *z = base + (VMR ? (int64_t)(2 * p) * G : 0);
    const int count = nrow * n;
    int l = threadIdx.x / n, k = threadIdx.x - l * n;
    const int dl = kCT / n, dk = kCT - dl * n;
    for (int e = threadIdx.x; e < count; e += kCT) {
      cp_async16(dst + k * PN + l, z + e);
      if (VMR) cp_async16(dst + k * PN + rt + l, z + G + e);
      l += dl;
      k += dk;
      if (k >= n) k -= n, ++l;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int cur = 0;
  load(p0, buf[0]);
  for (int p = p0; p < p1; ++p) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // stage i reads one buffer and writes the other; the results lie in the buffer the last one wrote
    const int total = ax.nst + (ax.R > 1 ? 1 : 0);
    const int res = ((total + ax.generic_first) & 1) ? 1 - cur : cur;
    double2 *dst = buf[res], *src = buf[cur];
    chunk_transform(
        ax, t, buf[1 - cur], buf[cur], PN, [&](int l) { return (const double2 *)src + l; },
        [](const double2 *q) { return *q; }, false,
        [&](int, double &c) {
          c = 1.0;
          return (const double *)nullptr;
        },
        [&](int l, int pos, double2 v) { dst[pos * PN + l] = v; });
    __syncthreads();
    cur = 1 - res;
    if (p + 1 < p1) load(p + 1, buf[cur]);
    const int count = nrow * n;
    int l = threadIdx.x / n, k = threadIdx.x - l * n;
    const int dl = kCT / n, dk = kCT - dl * n;
    if constexpr (VMR) {
      const int b = b0 + 2 * p;
      double *xa = out + ((int64_t)blockIdx.z * nboot + b) * G + (int64_t)row0 * n;
      for (int e = threadIdx.x; e < count; e += kCT) {
        const double2 z = dst[k * PN + l], w = dst[k * PN + rt + l];
        __stcg(xa + e, chunk_vmr(z.x, w.x, inv_n));
        if (b + 1 < nboot) __stcg(xa + G + e, chunk_vmr(z.y, w.y, inv_n));
        l += dl;
        k += dk;
        if (k >= n) k -= n, ++l;
      }
    } else {
      for (int e = threadIdx.x; e < count; e += kCT) {
        const double2 z = dst[k * PN + l];
        out[(int64_t)blockIdx.z * G + (int64_t)row0 * n + e] = sqrt(__fma_rn(z.x, z.x, __dmul_rn(z.y, z.y)));
        l += dl;
        k += dk;
        if (k >= n) k -= n, ++l;
      }
    }
  }
}

// Welford over the bootstraps in order, then f = log(scaled variance), of every point of C steps.
__global__ void __launch_bounds__(kCT) chunk_var_kernel(int64_t G, int nboot, const double *__restrict__ x,
                                                        const double *__restrict__ vscale, double *__restrict__ f) {
  __shared__ double recip[1024];  // 1 / i, IEEE
  const int64_t i = blockIdx.x * (int64_t)kCT + threadIdx.x;
  const double *p = x + (int64_t)blockIdx.y * nboot * G + i;
  double mean = 0.0, m2 = 0.0;
  for (int b0 = 0; b0 < nboot; b0 += 1024) {
    const int nb = min(1024, nboot - b0);
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += kCT) recip[b] = 1.0 / (double)(b0 + b + 1);
    __syncthreads();
    if (i < G) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) {
        const double v = __ldcg(p + (int64_t)(b0 + b) * G);
        const double delta = __dsub_rn(v, mean);
        mean = __fma_rn(delta, recip[b], mean);
        m2 = __fma_rn(delta, __dsub_rn(v, mean), m2);
      }
    }
  }
  if (i < G) {
    const double v = __ddiv_rn(__dmul_rn(vscale[blockIdx.y], m2), (double)(nboot - 1));
    f[(int64_t)blockIdx.y * G + i] = isfinite(v) ? log(v) : nan("");
  }
}

// The convergence state machine over the C steps of a chunk from s0 on, state in memory.
__global__ void __launch_bounds__(kCT) chunk_converge_kernel(int64_t G, int C, int s0, const double *__restrict__ f,
                                                             const double *__restrict__ mu,
                                                             const double *__restrict__ dlogt, double eps,
                                                             int64_t steps_low, int64_t steps_over, StepState cs) {
  const int64_t i = blockIdx.x * (int64_t)kCT + threadIdx.x;
  if (i >= G) return;
  double f1 = cs.f1[i], f2 = cs.f2[i], minimum = cs.minima[i], m = 0.0;
  uint16_t c_low = cs.c_low[i], c_over = cs.c_over[i];
  uint8_t flag = cs.flags[i];
  for (int c = 0; c < C; ++c) {
    const double fc = f[(int64_t)c * G + i];
    m = mu[(int64_t)c * G + i];
    const StabilityResult r =
        find_stability(fc, f1, f2, dlogt[s0 + c], eps, steps_low, steps_over, minimum, c_low, c_over, flag);
    c_low = r.c_low;
    c_over = r.c_over;
    flag = r.flag;
    minimum = r.new_min;
    if (r.more_stable) {
      cs.density[i] = m;
      cs.selected[i] = s0 + c;
    }
    f2 = f1;
    f1 = fc;
  }
  cs.f1[i] = f1;
  cs.f2[i] = f2;
  cs.minima[i] = minimum;
  cs.c_low[i] = c_low;
  cs.c_over[i] = c_over;
  cs.flags[i] = flag;
  cs.mu_last[i] = m;
}

// Lines per tile: as many as 2048 points hold, balanced over the tiles.
ChunkTile make_tile(int n, int R, int64_t lines, int most, bool odd) {
  const int64_t tiles = (lines + most - 1) / most;
  ChunkTile t;
  t.L = (int)((lines + tiles - 1) / tiles);
  t.Lr = t.L * R;
  t.P = odd ? t.Lr | 1 : t.Lr;
  t.PN = odd ? t.L | 1 : t.L;
  t.size = std::max(n * t.PN, n / R * t.P);
  t.dL = make_fastdiv((uint32_t)t.L);
  t.dLr = make_fastdiv((uint32_t)t.Lr);
  return t;
}

struct ChunkShape {
  int C, g;       // steps and pairs per chunk
  bool all_steps; // f and the means of every step are kept, the convergence walk runs once
};

// Chunks hold about 48 MB of intermediates (half of the L2 beside the spectra and the x
// values being written); f and means of all steps are kept up to 512 MB.
constexpr int64_t kChunkBytes = int64_t(48) << 20, kKeepBytes = int64_t(512) << 20;
ChunkShape chunk_shape(int64_t G, int npairs, int S) {
  ChunkShape c;
  const int64_t step = (int64_t)sizeof(double2) * (2 * npairs + 1) * G;
  c.C = (int)std::max<int64_t>(1, std::min<int64_t>(S, kChunkBytes / step));
  const int chunks = (S + c.C - 1) / c.C;
  c.C = (S + chunks - 1) / chunks;
  c.g = npairs;
  if (c.C == 1 && step > kChunkBytes) {
    c.g = (int)std::max<int64_t>(1, kChunkBytes / (2 * (int64_t)sizeof(double2) * G));
    const int groups = (npairs + c.g - 1) / c.g;
    c.g = (npairs + groups - 1) / groups;
  }
  c.all_steps = (int64_t)sizeof(double) * 2 * S * G <= kKeepBytes;
  return c;
}

}  // namespace

bool chunk_ok(const pkde_grid *g) {
  if (g->ndim < 2) return false;
  const int64_t G = grid_size(g);
  if (G > (int64_t(1) << 28)) return false;
  bool any = false;
  for (int j = 0; j < g->ndim; ++j) {
    const EngineAxis k = engine_axis(g, j);
    if (g->dims[j] > 1024 || !k.ok) return false;
    if (!k.pow2 && k.R == 1) {
      any = true;
      if (!stages_ok((int)g->dims[j])) return false;
    }
  }
  return any || getenv("PKDE_PROBE_CHUNK");
}

// Scratch: [intermediates][x][f][means].
static void chunk_scratch(int64_t G, int npairs, int nboot, int S, const ChunkShape &c, size_t off[5]) {
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  const int64_t arrays = std::max<int64_t>(c.g == npairs ? 2 * npairs + 1 : 2 * c.g, 1);
  const int64_t keep = c.all_steps ? S : c.C;
  off[0] = 0;
  off[1] = off[0] + al(sizeof(double2) * (size_t)(c.C * arrays * G));
  off[2] = off[1] + al(sizeof(double) * (size_t)((int64_t)c.C * nboot * G));
  off[3] = off[2] + al(sizeof(double) * (size_t)(keep * G));
  off[4] = off[3] + al(sizeof(double) * (size_t)(keep * G));
}

size_t chunk_scratch_bytes(const pkde_grid *g, int npairs, int nboot, int S) {
  const int64_t G = grid_size(g);
  size_t off[5];
  chunk_scratch(G, npairs, nboot, S, chunk_shape(G, npairs, S), off);
  return off[4];
}

bool chunk_keeps_all(const pkde_grid *g, int npairs, int S) { return chunk_shape(grid_size(g), npairs, S).all_steps; }

void run_chunk(pkde_ctx *ctx, const ChunkArgs &A, char *scratch, cudaStream_t st) {
  const pkde_grid *g = A.grid;
  const int N = g->ndim, S = A.S, nboot = A.nboot, npairs = A.npairs;
  const int G = (int)grid_size(g);
  const ChunkShape c = chunk_shape(G, npairs, S);
  size_t off[5];
  chunk_scratch(G, npairs, nboot, S, c, off);
  double2 *mid = (double2 *)(scratch + off[0]);
  double *x = (double *)(scratch + off[1]), *f = (double *)(scratch + off[2]), *mu = (double *)(scratch + off[3]);
  ChunkAxis ax[4];
  int inner = 1;
  for (int j = 0; j < N; ++j) {
    const EngineAxis k = engine_axis(g, j);
    ChunkAxis &a = ax[j];
    a = ChunkAxis{};
    a.n = (int)g->dims[j];
    a.R = k.R;
    a.M = a.n / a.R;
    a.inner = inner;
    a.lines = G / a.n;
    a.fused = k.pow2;
    a.twc = k.R > 1 ? combine_twiddles_device(ctx, k.R, a.M) : nullptr;
    a.nst = make_stages(ctx, a.M, a.st);
    a.generic_first = a.st[0].R > 5 && a.st[0].R != 8;
    inner *= a.n;
  }
  ChunkRun run{};
  run.N = N;
  run.G = G;
  run.mean = 2 * npairs;
  run.tab_stride = A.tab_stride;
  run.fz = A.fz;
  run.fw = A.fw;
  run.cw = A.cw;
  run.invG = 1.0 / (double)G;
  for (int j = 0; j < N; ++j) {
    run.dims[j] = (int)g->dims[j];
    run.aoff[j] = A.aoff[j];
  }
  // the passes over axes N..2 of `arrays` arrays from a0 in C steps from s0
  auto axes = [&](int64_t s0, int C, int a0, int arrays) {
    run.s0 = s0;
    run.C = C;
    run.a0 = a0;
    run.A = arrays;
    for (int j = N - 1; j >= 1; --j) {
      const ChunkAxis &a = ax[j];
      const int64_t lines = (int64_t)C * arrays * a.lines;
      const int most = kTilePts / a.n;
      ChunkTile t = make_tile(a.n, a.R, std::min<int64_t>(lines, most), most, false);
      const size_t smem = sizeof(double2) * (size_t)axis_tiles_held(a) * t.size + 32 * (size_t)t.L;
      const unsigned blocks = (unsigned)((lines + t.L - 1) / t.L);
      Trace tr(ctx, PKDE_PHASE_STEP_FFT, st);
      if (j == N - 1) {
        allow_dynamic_smem(ctx, chunk_axis_kernel<true>, smem);
        chunk_axis_kernel<true><<<blocks, kCT, smem, st>>>(a, t, run, A.spectra, mid);
      } else {
        allow_dynamic_smem(ctx, chunk_axis_kernel<false>, smem);
        chunk_axis_kernel<false><<<blocks, kCT, smem, st>>>(a, t, run, mid, mid);
      }
      PKDE_CHECK_LAUNCH();
    }
  };
  const ChunkAxis &a1 = ax[0];
  auto rows = [&](auto kern, int C, int arrays, int arr0, bool vmr, int pairs, int b0, double *out) {
    const int per = vmr ? 2 : 1;
    const int most = std::max(1, kTilePts / (per * a1.n));
    const ChunkTile rt = make_tile(a1.n, 1, a1.lines, most, false);
    ChunkTile t = make_tile(a1.n, a1.R, per * rt.L, per * rt.L, true);
    const size_t smem = sizeof(double2) * 2 * (size_t)t.size;
    const unsigned tiles = (unsigned)((a1.lines + rt.L - 1) / rt.L);
    // pairs per CTA: enough CTAs for a few waves, at most 8 pairs (the rows of the next pair are
    // fetched while this one's ratios are computed)
    int np = 1;
    if (vmr) {
      np = (int)std::max<int64_t>(1, std::min<int64_t>(8, (int64_t)tiles * C * pairs / (6 * 3 * ctx->sm_count)));
      const int parts = (pairs + np - 1) / np;
      np = (pairs + parts - 1) / parts;
    }
    allow_dynamic_smem(ctx, kern, smem);
    Trace tr(ctx, vmr ? PKDE_PHASE_STEP_VMR : PKDE_PHASE_STEP_MEANS, st);
    kern<<<dim3(tiles, vmr ? (unsigned)((pairs + np - 1) / np) : 1u, (unsigned)C), kCT, smem, st>>>(
        a1, t, G, arrays, arr0, rt.L, pairs, np, b0, nboot, A.inv_n, mid, out);
    PKDE_CHECK_LAUNCH();
  };
  for (int64_t s0 = 0; s0 < S; s0 += c.C) {
    const int C = (int)std::min<int64_t>(c.C, S - s0);
    double *fs = f + (c.all_steps ? s0 * G : 0), *ms = mu + (c.all_steps ? s0 * G : 0);
    if (c.g == npairs) {
      axes(s0, C, 0, 2 * npairs + 1);
      rows(chunk_rows_kernel<true>, C, 2 * npairs + 1, 0, true, npairs, 0, x);
      rows(chunk_rows_kernel<false>, C, 2 * npairs + 1, 2 * npairs, false, 0, 0, ms);
    } else {
      for (int p0 = 0; p0 < npairs; p0 += c.g) {
        const int np = std::min(c.g, npairs - p0);
        axes(s0, C, 2 * p0, 2 * np);
        rows(chunk_rows_kernel<true>, C, 2 * np, 0, true, np, 2 * p0, x);
      }
      axes(s0, C, 2 * npairs, 1);
      rows(chunk_rows_kernel<false>, C, 1, 0, false, 0, 0, ms);
    }
    {
      Trace tr(ctx, PKDE_PHASE_STEP_VMR, st);
      chunk_var_kernel<<<dim3((unsigned)((G + kCT - 1) / kCT), (unsigned)C), kCT, 0, st>>>(G, nboot, x, A.vscale + s0, fs);
    }
    PKDE_CHECK_LAUNCH();
    if (!c.all_steps) {
      Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
      chunk_converge_kernel<<<(unsigned)((G + kCT - 1) / kCT), kCT, 0, st>>>(
          G, C, (int)s0, fs, ms, A.dlogt, A.eps, A.steps_low, A.steps_over, A.cs);
    }
    PKDE_CHECK_LAUNCH();
  }
  if (c.all_steps) converge_steps(ctx, G, S, f, mu, A.dlogt, A.eps, A.steps_low, A.steps_over, A.cs, st);
}

}  // namespace pkde
