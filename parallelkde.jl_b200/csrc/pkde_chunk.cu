// Bandwidth steps of N-D estimations (N >= 2) several steps at a time: one launch per pass
// for a chunk of steps.
//
//   chunk_axis_kernel   inverse FFT along axes N..2, the propagation factors applied on
//                       the first load (FourierSpace.jl:215-262, :445-524);
//   chunk_rows_kernel   inverse FFT along axis 1 of the z and w rows of the pairs in turn, the
//                       variance-to-mean ratio of each bootstrap and its running variance
//                       (DirectSpace.jl:544-581), or of the means' rows (:747-764);
//   then the convergence walk (:829-1031), over all steps at the end where f and the
//   means of every step fit in memory, else chunk by chunk.
//
// The steps are independent given the spectra, so a chunk has no ordering inside it: the
// launches need no dependency counters, and every axis length fills its tiles (2048
// points, as many lines as fit, lines of different arrays and steps side by side).
// These kernels take any length; powers of two (pkde_chunk_pow2.cu) and other 2^a 3^b 5^c lengths
// (pkde_chunk_len.cuh) have their own.  The persistent engine (pkde_engine.cu) keeps longer axes.
#include <algorithm>
#include <cstring>

#include "pkde_chunk.cuh"
#include "pkde_jobs.cuh"
#include "pkde_tile.cuh"

namespace pkde {
namespace {

constexpr int kCT = 256;           // threads
constexpr int kTilePts = 8 * kCT;  // points per tile
constexpr int kCtas = 768 / kCT;   // CTAs per SM (80 registers a thread)
// Row kernel: tiles of 4 points a thread (and their z and w), 128 threads where a row fits, else
// 256 (384 x 384, 33 bootstraps, 40 steps: 5.2 ms with 128 threads, 5.8 with 256).
constexpr int kRowPts = 4;
constexpr int row_threads(int n) { return n <= 128 * kRowPts ? 128 : 256; }
constexpr int row_ctas(int T) { return 640 / T; }  // CTAs per SM (96 or 128 registers a thread)

// Tiles an axis pass holds: the first stage reads global memory and the last one writes it.
__host__ __device__ __forceinline__ int axis_tiles_held(const ChunkAxis &ax) {
  const int exchanges = ax.nst + (ax.R > 1 ? 1 : 0) - 1 + ax.generic_first;
  return exchanges < 2 ? exchanges : 2;
}

extern __shared__ double2 smc[];

// Where a tile's lines come from and go to, as byte offsets of 32 bits from a base that is the
// same for the block.
//   Src: at(l): offset of line l; load(offset); STEP(): bytes from element to element
//   Dst: at(l): offset (ok(offset): the line exists); store(offset, v); step()
// Lines through every stage, tiles a and b (byte addresses) in turn.  SCALED: element k of line
// l is multiplied by f[k] c, (f, c) = src.factor(l).  tw: the plain twiddle table in shared
// memory (copy_table), 0 where the line has none.  Every thread calls; the caller
// synchronises before the tiles are reused.
template <int T, bool SCALED, class Src, class Dst>
__device__ __forceinline__ void chunk_transform(const ChunkAxis &ax, const ChunkTile &t, unsigned a, unsigned b,
                                                unsigned tw, const Src &src, const Dst &dst) {
  const int R = ax.R, L = t.L, Lr = t.Lr, total = ax.nst + (R > 1 ? 1 : 0);
  const unsigned PB = t.P * 16u;
  const FastDiv dLr = t.dLr;
  auto put = [&](int l, int pos, int step, auto &v, auto rc) {  // elements pos + q step of line l
    constexpr int Q = decltype(rc)::value;
    const unsigned o = dst.at(l);
    if (dst.ok(o)) {
      unsigned p = o + pos * dst.step();
      const unsigned d = step * dst.step();
#pragma unroll
      for (int q = 0; q < Q; ++q, p += d) dst.store(p, v[q]);
    }
  };
  unsigned in = b, out = a;
  int i0 = 0;
  if (ax.generic_first) {  // its inputs pass through the tile (R = 1)
    for (int e = threadIdx.x; e < ax.n * L; e += T) {
      const int k = (int)fdiv((uint32_t)e, t.dL), l = e - k * L;
      double2 v = src.load(src.at(l) + k * src.step());
      if constexpr (SCALED) {
        double c;
        const double *f = src.factor(l, c);
        const double sc = __ldg(f + k) * c;
        v = make_double2(__dmul_rn(v.x, sc), __dmul_rn(v.y, sc));
      }
      sts(out + k * PB + l * 16u, v);
    }
    __syncthreads();
  } else {
    const Stage1 s = ax.st[0];
    auto first = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      const int items = s.nb * Lr;
      const unsigned sub = src.step() * R, d = sub * s.nb;
      for (int e = threadIdx.x; e < items; e += T) {
        const int j = (int)fdiv((uint32_t)e, dLr), l = e - j * Lr;
        const int n1 = R > 1 ? (int)fdiv((uint32_t)l, t.dL) : 0, line = l - n1 * L;
        double2 v[Q];
        unsigned p = src.at(line) + n1 * src.step() + j * sub;
#pragma unroll
        for (int r = 0; r < Q; ++r, p += d) v[r] = src.load(p);
        bool done = false;
        if constexpr (SCALED) {
          double c, sc[Q];
          const double *f = src.factor(line, c) + n1 + j * R;
          const int fd = s.nb * R;
#pragma unroll
          for (int r = 0; r < Q; ++r, f += fd) sc[r] = __ldg(f) * c;
          if constexpr (Q == 8) {
            if (ax.fused) {
              dft8_scaled(v, sc);
              done = true;
            }
          }
          if (!done) {
#pragma unroll
            for (int r = 0; r < Q; ++r) v[r] = make_double2(__dmul_rn(v[r].x, sc[r]), __dmul_rn(v[r].y, sc[r]));
          }
        }
        if (!done) dft_r<Q>(v);
        if (total == 1) {
          put(l, j * Q, 1, v, rc);
        } else {
          unsigned o = out + j * Q * PB + l * 16u;
#pragma unroll
          for (int q = 0; q < Q; ++q, o += PB) sts(o, v[q]);
        }
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
    i0 = 1;
  }
  in = a;
  out = b;
  for (int i = i0; i < ax.nst; ++i) {
    const Stage1 s = ax.st[i];
    const bool last = i + 1 == total;
    auto stage = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      const int items = s.nb * Lr, Ns = s.Ns;
      const unsigned d = s.nb * PB, od = Ns * PB;
      for (int e = threadIdx.x; e < items; e += T) {
        const int j = (int)fdiv((uint32_t)e, dLr), l = e - j * Lr;
        const int jq = (int)fdiv((uint32_t)j, s.dns), k = j - jq * Ns;
        double2 v[Q];
        unsigned p = in + j * PB + l * 16u;
#pragma unroll
        for (int r = 0; r < Q; ++r, p += d) v[r] = lds(p);
        if (k > 0) {
          const double2 *w = s.tw + k * (Q - 1) - 1;
#pragma unroll
          for (int r = 1; r < Q; ++r) v[r] = cmul1(v[r], __ldg(w + r));
        }
        dft_r<Q>(v);
        const int pos = j + jq * Ns * (Q - 1);
        if (last) {
          put(l, pos, Ns, v, rc);
        } else {
          unsigned o = out + pos * PB + l * 16u;
#pragma unroll
          for (int q = 0; q < Q; ++q, o += od) sts(o, v[q]);
        }
      }
    };
    switch (s.R) {
      case 8: stage(std::integral_constant<int, 8>{}); break;
      case 4: stage(std::integral_constant<int, 4>{}); break;
      case 2: stage(std::integral_constant<int, 2>{}); break;
      case 3: stage(std::integral_constant<int, 3>{}); break;
      case 5: stage(std::integral_constant<int, 5>{}); break;
      default: {
        const unsigned base = in;
        auto ld = [base](unsigned p) { return lds(base + p); };
        auto put1 = [&](int l, int pos, double2 v) {
          if (last) {
            const unsigned o = dst.at(l);
            if (dst.ok(o)) dst.store(o + pos * dst.step(), v);
          } else {
            sts(out + pos * PB + l * 16u, v);
          }
        };
        if (tw) {
          line_stage_generic<T>(s, ax.n, L, t.H, t.dH, PB, [tw](unsigned o) { return lds(tw + o); }, ld, put1);
        } else {
          const char *g = reinterpret_cast<const char *>(s.tw);
          line_stage_generic<T>(s, ax.n, L, t.H, t.dH, PB,
                                [g](unsigned o) { return __ldg(reinterpret_cast<const double2 *>(g + o)); }, ld, put1);
        }
        break;
      }
    }
    if (!last) __syncthreads();
    const unsigned x = in;
    in = out;
    out = x;
  }
  if (R > 1) {
    auto combine = [&](auto rc) {
      constexpr int Q = decltype(rc)::value;
      const int M = ax.M, items = M * L;
      for (int e = threadIdx.x; e < items; e += T) {
        const int k2 = (int)fdiv((uint32_t)e, t.dL), l = e - k2 * L;
        double2 y[Q];
        unsigned p = in + k2 * PB + l * 16u;
#pragma unroll
        for (int n1 = 0; n1 < Q; ++n1, p += L * 16u) {
          y[n1] = lds(p);
          if (n1 > 0) y[n1] = combine_cmul(y[n1], __ldg(ax.twc + (n1 - 1) * M + k2));
        }
        dft_r<Q>(y);
        put(l, k2, M, y, rc);
      }
    };
    if (R == 3) combine(std::integral_constant<int, 3>{});
    else combine(std::integral_constant<int, 5>{});
  }
}

// A line with a stage of another radix reads n factors all the time, which the L1 left beside the
// tiles does not hold for long: up to kTableLen points they go to shared memory (beyond, they would
// cost a resident CTA).
constexpr int kTableLen = 512;
__host__ __device__ __forceinline__ int table_points(const ChunkAxis &ax) {
  return ax.plain && ax.n <= kTableLen ? ax.n : 0;
}
template <int T>
__device__ __forceinline__ unsigned copy_table(const ChunkAxis &ax, double2 *to) {
  if (!table_points(ax)) return 0;
  for (int i = threadIdx.x; i < ax.n; i += T) to[i] = __ldg(ax.plain + i);
  return smem_of(to);
}

// Inverse FFT along one axis >= 2 of A arrays in each of C steps.  Tile = L consecutive lines of
// a step's flattened (array, line) index; blocks run over the steps first, so that the steps of
// a chunk read the same spectra while they are in the L2.  SPECTRA: the first pass, from the
// spectra, with the factors of every axis and the array's scalar; else in place.
template <bool SPECTRA>
struct AxisSrc {
  const char *base;
  unsigned ss;
  const unsigned *off;
  const double *const *f;
  const double *c;
  __device__ __forceinline__ unsigned step() const { return ss; }
  __device__ __forceinline__ unsigned at(int l) const { return off[l]; }
  __device__ __forceinline__ double2 load(unsigned o) const {
    const double2 *p = reinterpret_cast<const double2 *>(base + o);
    return SPECTRA ? __ldg(p) : __ldcg(p);
  }
  __device__ __forceinline__ const double *factor(int l, double &cl) const {
    cl = c[l];
    return f[l];
  }
};
struct AxisDst {
  char *base;
  unsigned ss;
  const unsigned *off;
  int valid;
  __device__ __forceinline__ unsigned step() const { return ss; }
  __device__ __forceinline__ unsigned at(int l) const { return l < valid ? off[l] : 0xffffffffu; }
  __device__ __forceinline__ bool ok(unsigned o) const { return o != 0xffffffffu; }
  __device__ __forceinline__ void store(unsigned o, double2 v) const {
    __stcg(reinterpret_cast<double2 *>(base + o), v);
  }
};

template <bool SPECTRA>
__device__ __forceinline__ void axis_body(const AxisJob &job, unsigned block) {
  const ChunkAxis &ax = job.ax;
  const ChunkTile &t = job.t;
  const ChunkRun &run = job.run;
  double2 *table = smc + axis_tiles_held(ax) * t.size;
  const unsigned tw = copy_table<kCT>(ax, table);
  const double **sf = reinterpret_cast<const double **>(table + table_points(ax));
  double *sc = reinterpret_cast<double *>(sf + t.L);
  unsigned *off = reinterpret_cast<unsigned *>(sc + t.L);
  const unsigned G = run.G, lines = ax.lines, inner = ax.inner;
  const unsigned tile = block / (unsigned)run.C, c = block - tile * run.C;
  const unsigned w0 = tile * t.L, arr0 = w0 / lines, li0 = w0 - arr0 * lines;
  const int valid = (int)min((unsigned)t.L, (unsigned)run.A * lines - w0);
  for (int l = threadIdx.x; l < t.L; l += kCT) {
    unsigned arr = arr0, li = li0 + (l < valid ? l : 0);
    while (li >= lines) li -= lines, ++arr;
    const unsigned o = li / inner;
    off[l] = ((arr - arr0) * G + o * ax.n * inner + (li - o * inner)) * 16u;
    if (SPECTRA) {
      const int64_t s = run.s0 + c;
      const int ar = run.a0 + (int)arr;
      const bool second = ar != run.mean && (ar & 1);
      const double *tab = (second ? run.fw : run.fz) + s * run.tab_stride;
      double f = second ? run.invG * run.cw[s] : run.invG;
      for (int q = 0; q < run.N - 1; ++q) {
        const unsigned d = run.dims[q], up = li / d;
        f *= tab[run.aoff[q] + (li - up * d)];
        li = up;
      }
      sf[l] = tab + run.aoff[run.N - 1];
      sc[l] = f;
    }
  }
  __syncthreads();
  const int64_t base = (int64_t)(c * run.A + arr0) * G;
  const AxisSrc<SPECTRA> src{
      reinterpret_cast<const char *>(job.in + (SPECTRA ? (int64_t)(run.a0 + arr0) * G : base)), inner * 16u, off, sf, sc};
  const AxisDst dst{reinterpret_cast<char *>(job.out + base), inner * 16u, off, valid};
  const unsigned a = smem_of(smc);
  chunk_transform<kCT, SPECTRA>(ax, t, a, a + t.size * 16u, tw, src, dst);
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

// The rows of a tile in shared memory, element k of line l at unit k PN + l.
struct RowsTile {
  unsigned base, ss;
  __device__ __forceinline__ unsigned step() const { return ss; }
  __device__ __forceinline__ unsigned at(int l) const { return base + l * 16u; }
  __device__ __forceinline__ bool ok(unsigned) const { return true; }
  __device__ __forceinline__ double2 load(unsigned o) const { return lds(o); }
  __device__ __forceinline__ void store(unsigned o, double2 v) const { sts(o, v); }
};

// Inverse FFT along axis 1 of rows [tile rt, + rt) of one step.  VMR: the z and w rows of the
// chunk's pairs in turn, line l < rt the z row l, line rt + l its w row, then the
// variance-to-mean ratio of both bootstraps of a pair and its running variance, a thread's
// points (at most kRowPts) in registers; the rows of the next pair come in by cp.async
// meanwhile.  After the last pair of the estimation f = log(scaled variance); between the
// groups of a step that is split the running (mean, m2) rests in memory.
// Else the rows of the means' array and their magnitudes.
template <int kRT, bool VMR>
__device__ __forceinline__ void rows_body(const RowsJob &job, unsigned block) {
  const ChunkAxis &ax = job.ax;
  const ChunkTile &t = job.t;
  const int G = job.G, rt = job.rt, nboot = job.nboot, n = ax.n;
  const unsigned bz = block / (unsigned)job.tiles, bx = block - bz * job.tiles;
  const unsigned PB = t.PN * 16u, tile0 = smem_of(smc), tsize = t.size * 16u;
  const int row0 = bx * rt, count = min(rt, ax.lines - row0) * n;
  const double2 *z = job.in + ((int64_t)bz * job.A + job.arr0) * G + (int64_t)row0 * n;
  // this thread's points e = threadIdx.x + q kRT of the tile: row l, element k at unit k PN + l
  unsigned at[kRowPts];
  {
    int l = threadIdx.x / n, k = threadIdx.x - l * n;
    const int dl = kRT / n, dk = kRT - dl * n;
#pragma unroll
    for (int q = 0; q < kRowPts; ++q) {
      at[q] = k * PB + l * 16u;
      l += dl;
      k += dk;
      if (k >= n) k -= n, ++l;
    }
  }
  auto load = [&](unsigned tile) {
#pragma unroll
    for (int q = 0; q < kRowPts; ++q) {
      const int e = threadIdx.x + q * kRT;
      if (e < count) {
        cp_async16(tile + at[q], z + e);
        if (VMR) cp_async16(tile + at[q] + rt * 16u, z + G + e);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int64_t o0 = (int64_t)bz * G + (int64_t)row0 * n;
  double2 st[VMR ? kRowPts : 1];
  if constexpr (VMR) {
#pragma unroll
    for (int q = 0; q < kRowPts; ++q) {
      const int e = threadIdx.x + q * kRT;
      st[q] = job.b0 > 0 && e < count ? job.state[o0 + e] : make_double2(0.0, 0.0);
    }
  }
  const int total = ax.nst + (ax.R > 1 ? 1 : 0) + ax.generic_first;
  unsigned cur = tile0;  // the tile (of two) that holds the inputs
  const unsigned both = 2 * tile0 + tsize;
  const unsigned tw = copy_table<kRT>(ax, smc + 2 * t.size);
  load(cur);
  const int pairs = VMR ? job.pairs : 1;
  for (int p = 0; p < pairs; ++p) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // each stage reads one tile and writes the other
    const unsigned res = (total & 1) ? both - cur : cur;
    chunk_transform<kRT, false>(ax, t, both - cur, cur, tw, RowsTile{cur, PB}, RowsTile{res, PB});
    __syncthreads();
    cur = both - res;
    z += 2 * (int64_t)G;
    if (p + 1 < pairs) load(cur);
    if constexpr (VMR) {
      const int b = job.b0 + 2 * p;
      const double ra = recip_of(job.recip, b + 1), rb = recip_of(job.recip, b + 2);
      const bool has_b = b + 1 < nboot;
#pragma unroll
      for (int q = 0; q < kRowPts; ++q) {
        if (threadIdx.x + q * kRT < count) {
          const double2 zv = lds(res + at[q]), wv = lds(res + at[q] + rt * 16u);
          double xa, xb;
          chunk_vmr2(zv, wv, job.inv_n, st[q].x, xa, xb);
          chunk_welford(xa, ra, st[q]);
          if (has_b) chunk_welford(xb, rb, st[q]);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < kRowPts; ++q) {
        const int e = threadIdx.x + q * kRT;
        if (e < count) {
          const double2 zv = lds(res + at[q]);
          job.out[o0 + e] = sqrt(__fma_rn(zv.x, zv.x, __dmul_rn(zv.y, zv.y)));
        }
      }
    }
  }
  if constexpr (VMR) {
    const bool done = job.b0 + 2 * pairs >= nboot;
    const double vs = job.vscale[bz], bm1 = (double)(nboot - 1);
#pragma unroll
    for (int q = 0; q < kRowPts; ++q) {
      const int e = threadIdx.x + q * kRT;
      if (e < count) {
        if (done) {
          const double v = __ddiv_rn(__dmul_rn(vs, st[q].y), bm1);
          job.out[o0 + e] = isfinite(v) ? log(v) : nan("");
        } else {
          job.state[o0 + e] = st[q];
        }
      }
    }
  }
}

template <int T, bool VMR>
__global__ void __launch_bounds__(T, row_ctas(T)) chunk_rows_kernel(const __grid_constant__ RowsJob job) {
  rows_body<T, VMR>(job, blockIdx.x);
}
template <int T, bool VMR>
__global__ void __launch_bounds__(T, row_ctas(T))
    chunk_rows_many_kernel(const RowsJob *jobs, const unsigned *block0, int count) {
  __shared__ RowsJob job;
  unsigned first;
  find_job(jobs, block0, count, job, first);
  rows_body<T, VMR>(job, blockIdx.x - first);
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

// Lines per tile, at most `most` (as many as its points hold) of `per` sub-tiles each (the rows
// kernel's z and w): the number that leaves the fewest butterfly slots of T threads empty over
// all tiles.  An item of a radix other than 2, 3, 4, 5, 8 is four outputs of R terms, so an idle
// third of a pass of threads costs as much as the other stages together (41 points, 256 threads: 49
// lines are 539 items in three passes, 46 are 506 in two: 150 x 77, 100 bootstraps, 250 steps 8.3 -> 7.9 ms).
int balanced_lines(const ChunkAxis &ax, int64_t lines, int most, int per, int T) {
  int best = 1;
  double best_cost = 1e300;
  for (int L = (int)std::min<int64_t>(most, lines); L >= 1 && 2 * L >= std::min<int64_t>(most, lines); --L) {
    double cost = 0.0;
    auto add = [&](int64_t items, double work) { cost += (double)((items + T - 1) / T) * work; };
    for (int i = 0; i < ax.nst; ++i) {
      const int R = ax.st[i].R, nb = ax.st[i].nb * ax.R;
      if (R <= 5 || R == 8) add((int64_t)nb * L * per, 12.0 * R);
      else add((int64_t)((R + 3) / 4) * nb * ((L * per + 1) / 2), 60.0 * R);
    }
    if (ax.R > 1) add((int64_t)ax.M * L * per, 12.0 * ax.R);
    cost *= (double)((lines + L - 1) / L);
    if (cost < best_cost) best_cost = cost, best = L;
  }
  return best;
}

ChunkTile make_tile(int n, int R, int L, bool odd) {
  ChunkTile t;
  t.L = L;
  t.Lr = t.L * R;
  t.P = odd ? t.Lr | 1 : t.Lr;
  t.PN = odd ? t.L | 1 : t.L;
  t.size = std::max(n * t.PN, n / R * t.P);
  t.H = (t.L + 1) / 2;
  t.dL = make_fastdiv((uint32_t)t.L);
  t.dH = make_fastdiv((uint32_t)t.H);
  t.dLr = make_fastdiv((uint32_t)t.Lr);
  return t;
}

struct ChunkShape {
  int C, g;       // steps and pairs per chunk
  bool all_steps; // f and the means of every step are kept, the convergence walk runs once
};

// Intermediates of a chunk and f and means of all steps are held up to these many bytes.  The
// larger the chunk the fewer launches drain the SMs, and the more steps share a reading of the
// spectra; that its intermediates leave the L2 costs less (100 x 100, 100 bootstraps, 250 steps, with
// 64 MB / 256 MB / 1 GB / 8 GB: 9.5 / 6.9 / 4.9 / 4.7 ms; 512 x 512, 64, 200, 1 / 2 / 4 / 8 GB: 45.2 / 41.3 /
// 40.0 / 39.7; 128^3, 32, 150: 194 / 193 / 173 / 167; 256 MB: 53 and 202).  Level kServeLevel for serving lanes, whose memory
// admission counts on it; a higher one where the device has no room or the caller's cap
// leaves none.
constexpr int64_t kMB = int64_t(1) << 20;
constexpr int64_t kChunkBytes[kChunkLevels] = {8192 * kMB, 2048 * kMB, 1024 * kMB, 256 * kMB, 16 * kMB};
constexpr int64_t kKeepBytes[kChunkLevels] = {8192 * kMB, 2048 * kMB, 512 * kMB, 128 * kMB, 4 * kMB};
ChunkShape chunk_shape(int64_t G, int npairs, int S, int level) {
  ChunkShape c;
  const int64_t step = (int64_t)sizeof(double2) * (2 * npairs + 1) * G;
  c.C = (int)std::max<int64_t>(1, std::min<int64_t>(S, kChunkBytes[level] / step));
  const int chunks = (S + c.C - 1) / c.C;
  c.C = (S + chunks - 1) / chunks;
  c.g = npairs;
  if (c.C == 1 && step > kChunkBytes[level]) {
    c.g = (int)std::max<int64_t>(1, kChunkBytes[level] / (2 * (int64_t)sizeof(double2) * G));
    const int groups = (npairs + c.g - 1) / c.g;
    c.g = (npairs + groups - 1) / groups;
  }
  c.all_steps = (int64_t)sizeof(double) * 2 * S * G <= kKeepBytes[level];
  return c;
}

}  // namespace

// Grids this path takes.  Against the persistent engine (whole calls, then here): its shared-memory
// tiles hold few lines of a length that is not 2^m, 3 2^m or 5 2^m (100 x 100, 100 bootstraps, 250
// steps: 67 ms, 3.6; 50 x 41 x 36, 32, 100: 149 and 8.7); its mixed-radix tiles leave a quarter of the
// threads idle (96^3, 32, 100: 100 and 51); on a small grid a step has too few tiles for its order
// of items (64 x 64, 33, 40: 1.8 and 0.33); on large powers of two it waits for dependencies and
// spills (512 x 512, 64, 200: 57.5 and 37.2; 128^3, 32, 150: 219 and 161).  It keeps axes of
// 1025 to 2048 points, and the contexts with a wait limit of their own.
bool chunk_ok(const pkde_grid *g) {
  if (g->ndim < 2) return false;
  const int64_t G = grid_size(g);
  if (G > (int64_t(1) << 26)) return false;  // byte offsets within a tile's arrays are 32 bits
  for (int j = 0; j < g->ndim; ++j) {
    const EngineAxis k = engine_axis(g, j);
    if (g->dims[j] > 1024 || !k.ok) return false;
    if (!k.pow2 && k.R == 1 && !stages_ok((int)g->dims[j])) return false;
  }
  return true;
}

// Scratch of one estimation: [intermediates][running variance][f][means].
static void chunk_scratch(int64_t G, int npairs, int S, const ChunkShape &c, size_t off[5]) {
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  const int64_t arrays = c.g == npairs ? 2 * npairs + 1 : 2 * c.g;
  const int64_t keep = c.all_steps ? S : c.C;
  off[0] = 0;
  off[1] = off[0] + al(sizeof(double2) * (size_t)(c.C * arrays * G));
  off[2] = off[1] + (c.g == npairs ? 0 : al(sizeof(double2) * (size_t)(c.C * G)));
  off[3] = off[2] + al(sizeof(double) * (size_t)(keep * G));
  off[4] = off[3] + al(sizeof(double) * (size_t)(keep * G));
}

size_t chunk_scratch_bytes(const pkde_grid *g, int npairs, int S, int level) {
  const int64_t G = grid_size(g);
  size_t off[5];
  chunk_scratch(G, npairs, S, chunk_shape(G, npairs, S, level), off);
  return off[4];
}

bool chunk_keeps_all(const pkde_grid *g, int npairs, int S, int level) {
  return chunk_shape(grid_size(g), npairs, S, level).all_steps;
}

namespace {

constexpr unsigned kSoloBlocks = 600;  // two waves of the general kernels

// One launch of a pass over the jobs of several estimations.
template <class J>
struct Launch {
  std::vector<J> jobs;
  std::vector<unsigned> block0;
  unsigned blocks = 0;
  size_t smem = 0;
  // jobs with a kernel for their length (chunk of steps of 96^3, 32 bootstraps, 100 steps: 69.5 ms in
  // the general kernels, 50.9; 100 x 100, 100, 250: 4.7 and 3.6), launched one by one: alone in
  // their pass, or large enough to fill the device
  std::vector<J> solo;
  void add(const J &j, unsigned n, size_t bytes, bool alone) {
    if ((j.ax.fused || j.ax.fixed) && (alone || n >= kSoloBlocks)) {
      solo.push_back(j);
      return;
    }
    jobs.push_back(j);
    block0.push_back(blocks);
    blocks += n;
    smem = std::max(smem, bytes);
  }
};
// The launches of chunk k: axis passes (first the one that reads the spectra), rows, variances.
struct ChunkLaunches {
  Launch<AxisJob> axis[3];
  Launch<RowsJob> vmr[2], means[2];  // 128 and 256 threads
};

struct ChunkPlan {
  ChunkAxis ax[4];
  ChunkRun run;
  ChunkShape c;
  double2 *mid;
  double2 *state;
  double *f, *mu;
  const double *recip;
};

const double *recip_table(pkde_ctx *ctx, cudaStream_t st) {
  DevBuf &b = ctx->chunk_recip;
  if (!b.ptr) {
    std::vector<double> r(kChunkRecip, 0.0);
    for (int i = 1; i < kChunkRecip; ++i) r[i] = 1.0 / (double)i;
    b.ensure(sizeof(double) * kChunkRecip);
    const cudaError_t e = cudaMemcpyAsync(b.ptr, r.data(), sizeof(double) * kChunkRecip, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) b.release();
    PKDE_CUDA_TRY(e);
  }
  return b.as<double>();
}

ChunkPlan plan_chunk(pkde_ctx *ctx, const ChunkArgs &A, char *scratch, cudaStream_t st) {
  ChunkPlan P{};
  const pkde_grid *g = A.grid;
  const int N = g->ndim, G = (int)grid_size(g);
  P.c = chunk_shape(G, A.npairs, A.S, A.level);
  P.recip = recip_table(ctx, st);
  size_t off[5];
  chunk_scratch(G, A.npairs, A.S, P.c, off);
  P.mid = (double2 *)(scratch + off[0]);
  P.state = (double2 *)(scratch + off[1]);
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
    a.twc = k.R > 1 ? combine_twiddles_device(ctx, k.R, a.M, st) : nullptr;
    a.nst = make_stages(ctx, a.M, a.st, st);
    a.fixed = chunk_len_known(a.n, a.R);
    for (int i = 0; i < a.nst; ++i)
      if (a.st[i].R > 5 && a.st[i].R != 8) a.plain = a.st[i].tw;
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
void add_axes(ChunkLaunches &L, const ChunkArgs &A, const ChunkPlan &P, int64_t s0, int C, int a0, int arrays,
              bool alone) {
  const int N = P.run.N;
  for (int j = N - 1; j >= 1; --j) {
    AxisJob J{};
    J.ax = P.ax[j];
    J.run = P.run;
    J.run.s0 = s0;
    J.run.C = C;
    J.run.a0 = a0;
    J.run.A = arrays;
    const int64_t lines = (int64_t)arrays * J.ax.lines;
    J.t = make_tile(J.ax.n, J.ax.R, balanced_lines(J.ax, lines, kTilePts / J.ax.n, 1, kCT), false);
    J.in = j == N - 1 ? A.spectra : P.mid;
    J.out = P.mid;
    const size_t smem = sizeof(double2) * (size_t)(axis_tiles_held(J.ax) * J.t.size + table_points(J.ax)) + 20 * (size_t)J.t.L;
    L.axis[N - 1 - j].add(J, (unsigned)((lines + J.t.L - 1) / J.t.L * C), smem, alone);
  }
}

void add_rows(Launch<RowsJob> (&Ls)[2], const ChunkArgs &A, const ChunkPlan &P, int64_t s0, int C, int arrays, int arr0,
              bool vmr, int pairs, int b0, double *out, bool alone) {
  RowsJob J{};
  J.ax = P.ax[0];
  const int per = vmr ? 2 : 1, T = row_threads(J.ax.n), most = T * kRowPts / J.ax.n;
  J.rt = balanced_lines(J.ax, J.ax.lines, most, per, T);
  J.t = make_tile(J.ax.n, J.ax.R, per * J.rt, true);
  J.G = P.run.G;
  J.A = arrays;
  J.arr0 = arr0;
  J.pairs = pairs;
  J.b0 = b0;
  J.nboot = A.nboot;
  J.inv_n = A.inv_n;
  J.vscale = A.vscale + s0;
  J.recip = P.recip;
  J.in = P.mid;
  J.state = P.state;
  J.out = out;
  J.tiles = (J.ax.lines + J.rt - 1) / J.rt;
  J.C = C;
  Ls[T == 128 ? 0 : 1].add(J, (unsigned)J.tiles * C, sizeof(double2) * (size_t)(2 * J.t.size + table_points(J.ax)), alone);
}

size_t al256c(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

// The bandwidth steps of `count` estimations, scratch[e] for each: chunk k of every
// estimation shares its launches.
void run_chunk(pkde_ctx *ctx, const ChunkArgs *args, int count, char *const *scratch, cudaStream_t st) {
  std::vector<ChunkPlan> plan;
  int chunks = 0;
  for (int e = 0; e < count; ++e) {
    plan.push_back(plan_chunk(ctx, args[e], scratch[e], st));
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
        add_axes(L, A, P, s0, C, 0, 2 * A.npairs + 1, count == 1);
        add_rows(L.vmr, A, P, s0, C, 2 * A.npairs + 1, 0, true, A.npairs, 0, fs, count == 1);
        add_rows(L.means, A, P, s0, C, 2 * A.npairs + 1, 2 * A.npairs, false, 0, 0, ms, count == 1);
      } else {
        for (int p0 = 0; p0 < A.npairs; p0 += P.c.g, ++at) {
          const int np = std::min(P.c.g, A.npairs - p0);
          ChunkLaunches &L = group(at);
          add_axes(L, A, P, s0, C, 2 * p0, 2 * np, count == 1);
          add_rows(L.vmr, A, P, s0, C, 2 * np, 0, true, np, 2 * p0, fs, count == 1);
        }
        ChunkLaunches &L = group(at);
        add_axes(L, A, P, s0, C, 2 * A.npairs, 1, count == 1);
        add_rows(L.means, A, P, s0, C, 1, 0, false, 0, 0, ms, count == 1);
      }
      if (!P.c.all_steps) converge[at].push_back({e, (int)s0});
    }
  }
  // job arrays to the device in one copy
  size_t bytes = 0;
  auto place = [&](auto &L) {
    const size_t at = bytes;
    if (L.jobs.size() < 2) return at;  // one job: a kernel parameter
    bytes += al256c(L.jobs.size() * sizeof(L.jobs[0])) + al256c(L.jobs.size() * sizeof(unsigned));
    return at;
  };
  std::vector<std::array<size_t, 7>> at(all.size());
  for (size_t i = 0; i < all.size(); ++i) {
    for (int j = 0; j < 3; ++j) at[i][j] = place(all[i].axis[j]);
    for (int j = 0; j < 2; ++j) {
      at[i][3 + j] = place(all[i].vmr[j]);
      at[i][5 + j] = place(all[i].means[j]);
    }
  }
  char *dev = bytes ? (char *)ensure(ctx, BUF_CHUNK, bytes) : nullptr;
  std::vector<char> host(bytes);
  auto store = [&](auto &L, size_t o) {
    if (L.jobs.size() < 2) return;
    std::memcpy(host.data() + o, L.jobs.data(), L.jobs.size() * sizeof(L.jobs[0]));
    std::memcpy(host.data() + o + al256c(L.jobs.size() * sizeof(L.jobs[0])), L.block0.data(),
                L.block0.size() * sizeof(unsigned));
  };
  for (size_t i = 0; i < all.size(); ++i) {
    for (int j = 0; j < 3; ++j) store(all[i].axis[j], at[i][j]);
    for (int j = 0; j < 2; ++j) {
      store(all[i].vmr[j], at[i][3 + j]);
      store(all[i].means[j], at[i][5 + j]);
    }
  }
  if (bytes) PKDE_CUDA_TRY(cudaMemcpyAsync(dev, host.data(), bytes, cudaMemcpyHostToDevice, st));
  auto launch = [&](auto &L, size_t o, int threads, int phase, auto one, auto many, auto solo) {
    for (const auto &j : L.solo) solo(j);
    if (L.jobs.empty()) return;
    using J = std::decay_t<decltype(L.jobs[0])>;
    const J *jobs = reinterpret_cast<const J *>(dev + o);
    const unsigned *block0 = reinterpret_cast<const unsigned *>(dev + o + al256c(L.jobs.size() * sizeof(J)));
    {
      Trace tr(ctx, phase, st);
      if (L.jobs.size() == 1) {
        allow_dynamic_smem(ctx, one, L.smem);
        one<<<L.blocks, threads, L.smem, st>>>(L.jobs[0]);
      } else {
        allow_dynamic_smem(ctx, many, L.smem);
        many<<<L.blocks, threads, L.smem, st>>>(jobs, block0, (int)L.jobs.size());
      }
    }
    PKDE_CHECK_LAUNCH();
  };
  for (size_t i = 0; i < all.size(); ++i) {
    ChunkLaunches &L = all[i];
    launch(L.axis[0], at[i][0], kCT, PKDE_PHASE_STEP_FFT, chunk_axis_kernel<true>, chunk_axis_many_kernel<true>,
           [&](const AxisJob &J) { (J.ax.fused ? chunk_pow2_axis : chunk_len_axis)(ctx, J, true, st); });
    for (int j = 1; j < 3; ++j)
      launch(L.axis[j], at[i][j], kCT, PKDE_PHASE_STEP_FFT, chunk_axis_kernel<false>, chunk_axis_many_kernel<false>,
             [&](const AxisJob &J) { (J.ax.fused ? chunk_pow2_axis : chunk_len_axis)(ctx, J, false, st); });
    auto solo_rows = [&](const RowsJob &J) { (J.ax.fused ? chunk_pow2_rows : chunk_len_rows)(ctx, J, st); };
    auto solo_means = [&](const RowsJob &J) { (J.ax.fused ? chunk_pow2_means : chunk_len_means)(ctx, J, st); };
    launch(L.vmr[0], at[i][3], 128, PKDE_PHASE_STEP_VMR, chunk_rows_kernel<128, true>, chunk_rows_many_kernel<128, true>,
           solo_rows);
    launch(L.vmr[1], at[i][4], 256, PKDE_PHASE_STEP_VMR, chunk_rows_kernel<256, true>, chunk_rows_many_kernel<256, true>,
           solo_rows);
    launch(L.means[0], at[i][5], 128, PKDE_PHASE_STEP_MEANS, chunk_rows_kernel<128, false>,
           chunk_rows_many_kernel<128, false>, solo_means);
    launch(L.means[1], at[i][6], 256, PKDE_PHASE_STEP_MEANS, chunk_rows_kernel<256, false>,
           chunk_rows_many_kernel<256, false>, solo_means);
    for (const auto &c : converge[i]) {
      const ChunkArgs &A = args[c[0]];
      const ChunkPlan &P = plan[c[0]];
      Trace tr(ctx, PKDE_PHASE_STEP_MEANS, st);
      chunk_converge_kernel<<<(unsigned)((P.run.G + kCT - 1) / kCT), kCT, 0, st>>>(
          P.run.G, std::min(P.c.C, A.S - c[1]), c[1], P.f, P.mu, A.dlogt, A.eps, A.steps_low, A.steps_over, A.cs);
    }
    PKDE_CHECK_LAUNCH();
  }
  std::vector<ConvergeJob> walks;
  for (int e = 0; e < count; ++e) {
    const ChunkArgs &A = args[e];
    if (plan[e].c.all_steps)
      walks.push_back({plan[e].run.G, A.steps_low, A.steps_over, plan[e].f, plan[e].mu, A.dlogt, A.eps, A.S, A.cs});
  }
  converge_steps(ctx, walks, st);
}

}  // namespace pkde
