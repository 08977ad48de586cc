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
#include <cstring>

#include "pkde_lines.cuh"
#include "pkde_step.cuh"

namespace pkde {
namespace {

constexpr int kCT = 256;           // threads
constexpr int kTilePts = 8 * kCT;  // points per tile
constexpr int kCtas = 768 / kCT;   // CTAs per SM (80 registers a thread)

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

// A launch covers one or several estimations: blocks [block0, next job's block0) are the job's.
struct AxisJob {
  ChunkAxis ax;
  ChunkTile t;
  ChunkRun run;
  const double2 *in;
  double2 *out;
};
struct RowsJob {
  ChunkAxis ax;
  ChunkTile t;
  int G, A, arr0, rt, pairs, np, b0, nboot, tiles, parts;  // blocks: tiles x parts x steps
  double inv_n;
  const double2 *in;
  double *out;
};
struct VarJob {
  int64_t G;
  int nboot, blocks;  // blocks: per step
  const double *x, *vscale;
  double *f;
};

// The job of this block: of several (job array and first blocks in device memory) copied into
// shared memory, of one the kernel's own parameter.
template <class J>
__device__ __forceinline__ void find_job(const J *jobs, const unsigned *block0, int count, J &sj, unsigned &first) {
  __shared__ int s_job;
  if (threadIdx.x < 32) {
    int job = 0;
    for (;;) {  // block0 increases: the lanes at or below this block form a prefix
      const int k = job + 1 + (int)threadIdx.x;
      const bool le = k < count && __ldg(block0 + k) <= blockIdx.x;
      const int c = __popc(__ballot_sync(0xffffffffu, le));
      job += c;
      if (c < 32) break;
    }
    if (threadIdx.x == 0) s_job = job;
  }
  __syncthreads();
  const int job = s_job;
  const int *src = reinterpret_cast<const int *>(jobs + job);
  int *dst = reinterpret_cast<int *>(&sj);
  for (int i = threadIdx.x; i < (int)(sizeof(J) / sizeof(int)); i += blockDim.x) dst[i] = __ldg(src + i);
  first = __ldg(block0 + job);
  __syncthreads();
}

// Lines through every stage: input element k of line l at src(l) + k ss (loaded by ld, scaled by
// scale(l) and f[k] where `scaled`), tiles a and b in turn, output position p of line l through
// st(l, p, value).  Every thread calls; the caller synchronises before the tiles are reused.
template <class Src, class Ld, class Fac, class St>
__device__ __forceinline__ void chunk_transform(const ChunkAxis &ax, const ChunkTile &t, int a, int b,
                                                int64_t ss, Src src, Ld ld, bool scaled, Fac fac, St st) {
  const int R = ax.R, L = t.L, Lr = t.Lr, P = t.P;
  const int total = ax.nst + (R > 1 ? 1 : 0);
  auto sub = [&](int l, int &n1) {  // sub-line l = n1 L + line
    n1 = R > 1 ? (int)fdiv((uint32_t)l, t.dL) : 0;
    return l - n1 * L;
  };
  int s0 = 0;
  int in = b, out = a;  // tiles, as units of smc (pointers would lose the address space)
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
      smc[out + k * P + l] = v;
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
          double2 *o = smc + out + pos * P + l;
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
        const double2 *p = smc + in + j * P + l;
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
          double2 *o = smc + out + pos * P + l;
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
        if (last) line_stage_generic<kCT>(s, ax.n, Lr, t.dLr, smc + in, P, st);
        else line_stage_generic<kCT>(s, ax.n, Lr, t.dLr, smc + in, P, [&](int l, int pos, double2 v) { smc[out + pos * P + l] = v; });
        break;
    }
    if (!last) __syncthreads();
    const int x = in;
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
          y[n1] = smc[in + k2 * P + n1 * L + l];
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
__device__ __forceinline__ void axis_body(const AxisJob &job, unsigned block) {
  const ChunkAxis &ax = job.ax;
  const ChunkTile &t = job.t;
  const ChunkRun &run = job.run;
  const double2 *in = job.in;
  double2 *out = job.out;
  int64_t *so = reinterpret_cast<int64_t *>(smc + axis_tiles_held(ax) * t.size);
  int64_t *si = so + t.L;
  const double **sf = reinterpret_cast<const double **>(si + t.L);
  double *sc = reinterpret_cast<double *>(sf + t.L);
  const int G = run.G;
  {
    const unsigned per = (unsigned)run.A * ax.lines, total = (unsigned)run.C * per;
    for (int l = threadIdx.x; l < t.L; l += kCT) {
      unsigned w = block * (unsigned)t.L + l;
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
      ax, t, 0, t.size, ax.inner, [&](int l) { return in + si[l]; },
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

template <bool SPECTRA>
__global__ void __launch_bounds__(kCT, kCtas) chunk_axis_kernel(const __grid_constant__ AxisJob job) {
  axis_body<SPECTRA>(job, blockIdx.x);
}
template <bool SPECTRA>
__global__ void __launch_bounds__(kCT, kCtas)
    chunk_axis_many_kernel(const AxisJob *jobs, const unsigned *block0, int count) {
  __shared__ AxisJob job;
  unsigned first;
  find_job(jobs, block0, count, job, first);
  axis_body<SPECTRA>(job, blockIdx.x - first);
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
__device__ __forceinline__ void rows_body(const RowsJob &job, unsigned block) {
  const ChunkAxis &ax = job.ax;
  const ChunkTile &t = job.t;
  const int G = job.G, rt = job.rt, nboot = job.nboot;
  const double inv_n = job.inv_n;
  const unsigned q = block / (unsigned)job.tiles, bx = block - q * job.tiles;
  const unsigned bz = q / (unsigned)job.parts, by = q - bz * job.parts;
  const int n = ax.n, PN = t.PN, row0 = bx * rt, nrow = min(rt, ax.lines - row0);
  const int p0 = VMR ? by * job.np : 0, p1 = VMR ? min(p0 + job.np, job.pairs) : 1;
  const double2 *base = job.in + ((int64_t)bz * job.A + job.arr0) * G + (int64_t)row0 * n;
  auto load = [&](int p, int tile) {
    double2 *dst = smc + tile;
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
  int cur = 0;  // the tile (of two) that holds the inputs
  load(p0, 0);
  for (int p = p0; p < p1; ++p) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // stage i reads one buffer and writes the other; the results lie in the buffer the last one wrote
    const int total = ax.nst + (ax.R > 1 ? 1 : 0);
    const int res = ((total + ax.generic_first) & 1) ? 1 - cur : cur;
    const int dst = res * t.size, src = cur * t.size;
    chunk_transform(
        ax, t, t.size - src, src, PN, [&](int l) { return (const double2 *)smc + src + l; },
        [](const double2 *q) { return *q; }, false,
        [&](int, double &c) {
          c = 1.0;
          return (const double *)nullptr;
        },
        [&](int l, int pos, double2 v) { smc[dst + pos * PN + l] = v; });
    __syncthreads();
    cur = 1 - res;
    if (p + 1 < p1) load(p + 1, cur * t.size);
    const int count = nrow * n;
    int l = threadIdx.x / n, k = threadIdx.x - l * n;
    const int dl = kCT / n, dk = kCT - dl * n;
    if constexpr (VMR) {
      const int b = job.b0 + 2 * p;
      double *xa = job.out + ((int64_t)bz * nboot + b) * G + (int64_t)row0 * n;
      for (int e = threadIdx.x; e < count; e += kCT) {
        const double2 z = smc[dst + k * PN + l], w = smc[dst + k * PN + rt + l];
        __stcg(xa + e, chunk_vmr(z.x, w.x, inv_n));
        if (b + 1 < nboot) __stcg(xa + G + e, chunk_vmr(z.y, w.y, inv_n));
        l += dl;
        k += dk;
        if (k >= n) k -= n, ++l;
      }
    } else {
      for (int e = threadIdx.x; e < count; e += kCT) {
        const double2 z = smc[dst + k * PN + l];
        job.out[(int64_t)bz * G + (int64_t)row0 * n + e] = sqrt(__fma_rn(z.x, z.x, __dmul_rn(z.y, z.y)));
        l += dl;
        k += dk;
        if (k >= n) k -= n, ++l;
      }
    }
  }
}

template <bool VMR>
__global__ void __launch_bounds__(kCT, kCtas) chunk_rows_kernel(const __grid_constant__ RowsJob job) {
  rows_body<VMR>(job, blockIdx.x);
}
template <bool VMR>
__global__ void __launch_bounds__(kCT, kCtas)
    chunk_rows_many_kernel(const RowsJob *jobs, const unsigned *block0, int count) {
  __shared__ RowsJob job;
  unsigned first;
  find_job(jobs, block0, count, job, first);
  rows_body<VMR>(job, blockIdx.x - first);
}

// Welford over the bootstraps in order, then f = log(scaled variance), of every point of the
// job's steps.
constexpr int kVT = 128;
__global__ void __launch_bounds__(kVT) chunk_var_kernel(const VarJob *jobs, const unsigned *block0, int count) {
  __shared__ VarJob J;
  __shared__ double recip[1024];  // 1 / i, IEEE
  unsigned first;
  find_job(jobs, block0, count, J, first);
  const int64_t G = J.G;
  const unsigned step = (blockIdx.x - first) / (unsigned)J.blocks;
  const int64_t i = (blockIdx.x - first - step * J.blocks) * (int64_t)kVT + threadIdx.x;
  const double *p = J.x + (int64_t)step * J.nboot * G + i;
  double mean = 0.0, m2 = 0.0;
  for (int b0 = 0; b0 < J.nboot; b0 += 1024) {
    const int nb = min(1024, J.nboot - b0);
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += kVT) recip[b] = 1.0 / (double)(b0 + b + 1);
    __syncthreads();
    if (i < G) {
#pragma unroll 16
      for (int b = 0; b < nb; ++b) {
        const double v = __ldcg(p + (int64_t)(b0 + b) * G);
        const double delta = __dsub_rn(v, mean);
        mean = __fma_rn(delta, recip[b], mean);
        m2 = __fma_rn(delta, __dsub_rn(v, mean), m2);
      }
    }
  }
  if (i < G) {
    const double v = __ddiv_rn(__dmul_rn(J.vscale[step], m2), (double)(J.nboot - 1));
    J.f[(int64_t)step * G + i] = isfinite(v) ? log(v) : nan("");
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

// Chunks hold up to 64 MB of intermediates (half of the L2 beside the spectra and the x
// values being written); f and means of all steps are kept up to 512 MB.
constexpr int64_t kChunkBytes = int64_t(64) << 20, kKeepBytes = int64_t(512) << 20;
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

// Grids with an axis that is neither a power of two nor 3 or 5 times one: the engine's
// shared-memory tiles hold few lines there (100 x 100, 100 bootstraps, 250 steps: 66 ms
// against 8.1 ms here; 50 x 41 x 36, 32 bootstraps, 100 steps: 148 against 16.6 ms).  Small grids of
// any lengths: a step has too few tiles for the engine's order of items (64 x 64, 33 bootstraps,
// 40 steps: 2.0 against 0.4 ms; 64^3: 7 against 11 ms).
constexpr int64_t kSmallGrid = 65536;
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
  return any || G < kSmallGrid;
}

// Scratch of one estimation: [intermediates][x][f][means].
static void chunk_scratch(int64_t G, int npairs, int nboot, int S, const ChunkShape &c, size_t off[5]) {
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  const int64_t arrays = c.g == npairs ? 2 * npairs + 1 : 2 * c.g;
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

namespace {

// One launch of a pass over the jobs of several estimations.
template <class J>
struct Launch {
  std::vector<J> jobs;
  std::vector<unsigned> block0;
  unsigned blocks = 0;
  size_t smem = 0;
  void add(const J &j, unsigned n, size_t bytes) {
    jobs.push_back(j);
    block0.push_back(blocks);
    blocks += n;
    smem = std::max(smem, bytes);
  }
};
// The launches of chunk k: axis passes (first the one that reads the spectra), rows, variances.
struct ChunkLaunches {
  Launch<AxisJob> axis[3];
  Launch<RowsJob> vmr, means;
  Launch<VarJob> var;
};

struct ChunkPlan {
  ChunkAxis ax[4];
  ChunkRun run;
  ChunkShape c;
  double2 *mid;
  double *x, *f, *mu;
};

ChunkPlan plan_chunk(pkde_ctx *ctx, const ChunkArgs &A, char *scratch) {
  ChunkPlan P{};
  const pkde_grid *g = A.grid;
  const int N = g->ndim, G = (int)grid_size(g);
  P.c = chunk_shape(G, A.npairs, A.S);
  size_t off[5];
  chunk_scratch(G, A.npairs, A.nboot, A.S, P.c, off);
  P.mid = (double2 *)(scratch + off[0]);
  P.x = (double *)(scratch + off[1]);
  P.f = (double *)(scratch + off[2]);
  P.mu = (double *)(scratch + off[3]);
  int inner = 1;
  for (int j = 0; j < N; ++j) {
    const EngineAxis k = engine_axis(g, j);
    ChunkAxis &a = P.ax[j];
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
  ChunkRun &run = P.run;
  run.N = N;
  run.G = G;
  run.mean = 2 * A.npairs;
  run.tab_stride = A.tab_stride;
  run.fz = A.fz;
  run.fw = A.fw;
  run.cw = A.cw;
  run.invG = 1.0 / (double)G;
  for (int j = 0; j < N; ++j) {
    run.dims[j] = (int)g->dims[j];
    run.aoff[j] = A.aoff[j];
  }
  return P;
}

// Passes over axes N..2 of `arrays` arrays from a0 in C steps from s0.
void add_axes(ChunkLaunches &L, const ChunkArgs &A, const ChunkPlan &P, int64_t s0, int C, int a0, int arrays) {
  const int N = P.run.N;
  for (int j = N - 1; j >= 1; --j) {
    AxisJob J{};
    J.ax = P.ax[j];
    J.run = P.run;
    J.run.s0 = s0;
    J.run.C = C;
    J.run.a0 = a0;
    J.run.A = arrays;
    const int64_t lines = (int64_t)C * arrays * J.ax.lines;
    const int most = kTilePts / J.ax.n;
    J.t = make_tile(J.ax.n, J.ax.R, std::min<int64_t>(lines, most), most, false);
    J.in = j == N - 1 ? A.spectra : P.mid;
    J.out = P.mid;
    const size_t smem = sizeof(double2) * (size_t)axis_tiles_held(J.ax) * J.t.size + 32 * (size_t)J.t.L;
    L.axis[N - 1 - j].add(J, (unsigned)((lines + J.t.L - 1) / J.t.L), smem);
  }
}

void add_rows(pkde_ctx *ctx, Launch<RowsJob> &L, const ChunkArgs &A, const ChunkPlan &P, int C, int arrays, int arr0,
              bool vmr, int pairs, int b0, double *out) {
  RowsJob J{};
  J.ax = P.ax[0];
  const int per = vmr ? 2 : 1, most = std::max(1, kTilePts / (per * J.ax.n));
  J.rt = make_tile(J.ax.n, 1, J.ax.lines, most, false).L;
  J.t = make_tile(J.ax.n, J.ax.R, per * J.rt, per * J.rt, true);
  J.G = P.run.G;
  J.A = arrays;
  J.arr0 = arr0;
  J.pairs = pairs;
  J.b0 = b0;
  J.nboot = A.nboot;
  J.inv_n = A.inv_n;
  J.in = P.mid;
  J.out = out;
  J.tiles = (J.ax.lines + J.rt - 1) / J.rt;
  // pairs per CTA: enough CTAs for a few waves, at most 8 pairs (the rows of the next pair are
  // fetched while this one's ratios are computed)
  J.np = 1;
  J.parts = 1;
  if (vmr) {
    J.np = (int)std::max<int64_t>(
        1, std::min<int64_t>(8, (int64_t)J.tiles * C * pairs / (6 * kCtas * (int64_t)ctx->sm_count)));
    J.parts = (pairs + J.np - 1) / J.np;
    J.np = (pairs + J.parts - 1) / J.parts;
  }
  L.add(J, (unsigned)J.tiles * J.parts * C, sizeof(double2) * 2 * (size_t)J.t.size);
}

size_t al256c(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

// The bandwidth steps of `count` estimations, scratch[e] for each: chunk k of every
// estimation shares its launches.
void run_chunk(pkde_ctx *ctx, const ChunkArgs *args, int count, char *const *scratch, cudaStream_t st) {
  std::vector<ChunkPlan> plan;
  int chunks = 0;
  for (int e = 0; e < count; ++e) {
    plan.push_back(plan_chunk(ctx, args[e], scratch[e]));
    chunks = std::max(chunks, (args[e].S + plan[e].c.C - 1) / plan[e].c.C);
  }
  // every launch of the call; estimations whose steps are split by pair groups add launches of their own
  std::vector<ChunkLaunches> all;
  std::vector<std::vector<std::array<int, 2>>> converge;  // per launch group: (estimation, first step)
  for (int k = 0; k < chunks; ++k) {
    const size_t g0 = all.size();
    all.emplace_back();
    converge.emplace_back();
    for (int e = 0; e < count; ++e) {
      const ChunkArgs &A = args[e];
      const ChunkPlan &P = plan[e];
      const int64_t G = P.run.G, s0 = (int64_t)k * P.c.C;
      if (s0 >= A.S) continue;
      const int C = (int)std::min<int64_t>(P.c.C, A.S - s0);
      double *fs = P.f + (P.c.all_steps ? s0 * G : 0), *ms = P.mu + (P.c.all_steps ? s0 * G : 0);
      size_t at = g0;
      auto group = [&](size_t i) -> ChunkLaunches & {
        while (all.size() <= i) {
          all.emplace_back();
          converge.emplace_back();
        }
        return all[i];
      };
      if (P.c.g == A.npairs) {
        ChunkLaunches &L = group(at);
        add_axes(L, A, P, s0, C, 0, 2 * A.npairs + 1);
        add_rows(ctx, L.vmr, A, P, C, 2 * A.npairs + 1, 0, true, A.npairs, 0, P.x);
        add_rows(ctx, L.means, A, P, C, 2 * A.npairs + 1, 2 * A.npairs, false, 0, 0, ms);
      } else {
        for (int p0 = 0; p0 < A.npairs; p0 += P.c.g, ++at) {
          const int np = std::min(P.c.g, A.npairs - p0);
          ChunkLaunches &L = group(at);
          add_axes(L, A, P, s0, C, 2 * p0, 2 * np);
          add_rows(ctx, L.vmr, A, P, C, 2 * np, 0, true, np, 2 * p0, P.x);
        }
        ChunkLaunches &L = group(at);
        add_axes(L, A, P, s0, C, 2 * A.npairs, 1);
        add_rows(ctx, L.means, A, P, C, 1, 0, false, 0, 0, ms);
      }
      VarJob V{};
      V.G = G;
      V.nboot = A.nboot;
      V.blocks = (int)((G + kVT - 1) / kVT);
      V.x = P.x;
      V.vscale = A.vscale + s0;
      V.f = fs;
      group(at).var.add(V, (unsigned)(V.blocks * C), 0);
      if (!P.c.all_steps) converge[at].push_back({e, (int)s0});
    }
  }
  // job arrays to the device in one copy
  size_t bytes = 0;
  auto place = [&](auto &L, bool always) {
    const size_t at = bytes;
    if (L.jobs.size() < 2 && !always) return at;  // one job: a kernel parameter
    bytes += al256c(L.jobs.size() * sizeof(L.jobs[0])) + al256c(L.jobs.size() * sizeof(unsigned));
    return at;
  };
  std::vector<std::array<size_t, 6>> at(all.size());
  for (size_t i = 0; i < all.size(); ++i) {
    for (int j = 0; j < 3; ++j) at[i][j] = place(all[i].axis[j], false);
    at[i][3] = place(all[i].vmr, false);
    at[i][4] = place(all[i].means, false);
    at[i][5] = place(all[i].var, true);
  }
  char *dev = (char *)ensure(ctx, BUF_CHUNK, bytes);
  std::vector<char> host(bytes);
  auto store = [&](auto &L, size_t o, bool always) {
    if (L.jobs.empty() || (L.jobs.size() < 2 && !always)) return;
    std::memcpy(host.data() + o, L.jobs.data(), L.jobs.size() * sizeof(L.jobs[0]));
    std::memcpy(host.data() + o + al256c(L.jobs.size() * sizeof(L.jobs[0])), L.block0.data(),
                L.block0.size() * sizeof(unsigned));
  };
  for (size_t i = 0; i < all.size(); ++i) {
    for (int j = 0; j < 3; ++j) store(all[i].axis[j], at[i][j], false);
    store(all[i].vmr, at[i][3], false);
    store(all[i].means, at[i][4], false);
    store(all[i].var, at[i][5], true);
  }
  PKDE_CUDA_TRY(cudaMemcpyAsync(dev, host.data(), bytes, cudaMemcpyHostToDevice, st));
  auto launch = [&](auto &L, size_t o, int phase, auto one, auto many) {
    if (L.jobs.empty()) return;
    using J = std::decay_t<decltype(L.jobs[0])>;
    const J *jobs = reinterpret_cast<const J *>(dev + o);
    const unsigned *block0 = reinterpret_cast<const unsigned *>(dev + o + al256c(L.jobs.size() * sizeof(J)));
    {
      Trace tr(ctx, phase, st);
      if (L.jobs.size() == 1) {
        allow_dynamic_smem(ctx, one, L.smem);
        one<<<L.blocks, kCT, L.smem, st>>>(L.jobs[0]);
      } else {
        allow_dynamic_smem(ctx, many, L.smem);
        many<<<L.blocks, kCT, L.smem, st>>>(jobs, block0, (int)L.jobs.size());
      }
    }
    PKDE_CHECK_LAUNCH();
  };
  for (size_t i = 0; i < all.size(); ++i) {
    ChunkLaunches &L = all[i];
    launch(L.axis[0], at[i][0], PKDE_PHASE_STEP_FFT, chunk_axis_kernel<true>, chunk_axis_many_kernel<true>);
    for (int j = 1; j < 3; ++j)
      launch(L.axis[j], at[i][j], PKDE_PHASE_STEP_FFT, chunk_axis_kernel<false>, chunk_axis_many_kernel<false>);
    launch(L.vmr, at[i][3], PKDE_PHASE_STEP_VMR, chunk_rows_kernel<true>, chunk_rows_many_kernel<true>);
    launch(L.means, at[i][4], PKDE_PHASE_STEP_MEANS, chunk_rows_kernel<false>, chunk_rows_many_kernel<false>);
    if (!L.var.jobs.empty()) {
      const char *o = dev + at[i][5];
      Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
      chunk_var_kernel<<<L.var.blocks, kVT, 0, st>>>(
          reinterpret_cast<const VarJob *>(o),
          reinterpret_cast<const unsigned *>(o + al256c(L.var.jobs.size() * sizeof(VarJob))), (int)L.var.jobs.size());
    }
    PKDE_CHECK_LAUNCH();
    for (const auto &c : converge[i]) {
      const ChunkArgs &A = args[c[0]];
      const ChunkPlan &P = plan[c[0]];
      Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
      chunk_converge_kernel<<<(unsigned)((P.run.G + kCT - 1) / kCT), kCT, 0, st>>>(
          P.run.G, std::min(P.c.C, A.S - c[1]), c[1], P.f, P.mu, A.dlogt, A.eps, A.steps_low, A.steps_over, A.cs);
    }
    PKDE_CHECK_LAUNCH();
  }
  for (int e = 0; e < count; ++e) {
    const ChunkArgs &A = args[e];
    if (plan[e].c.all_steps)
      converge_steps(ctx, plan[e].run.G, A.S, plan[e].f, plan[e].mu, A.dlogt, A.eps, A.steps_low, A.steps_over, A.cs, st);
  }
}

}  // namespace pkde
