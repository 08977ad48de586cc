// Binning of the estimators: every bootstrap resample and the samples themselves onto the
// grid (cloud in cell), into the layout of the paired spectra: array 2p holds the means of
// resamples 2p and 2p + 1 as real and imaginary part, array 2p + 1 their squares, the last
// one the samples.
//
// Reference: DirectSpace.jl:196-242 (generate_dirac_cpu!, the FP64 arithmetic followed
// here), :364-477, :479-512 (check_data).
//
// The samples are put in the order of their lower cells once (counting sort), each resample's
// draws become multiplicities per sample in that order, and the sums are taken over
// multiplicity x term.  Each of the 2^N corner terms of a sample is computed in FP64 as the
// reference's CPU path does and split into two fixed-point parts (the scaled term's nearest
// integer and its remainder scaled further), with exponents from the largest count of any
// cell, so that every sum is one of exact 64-bit integers: no order of the atomics, and no
// division of the work, changes a bit.
#include <algorithm>
#include <cstring>

#include "pkde_jobs.cuh"

namespace pkde {

struct BinJob {
  int N, samples;  // samples a warp takes in a row
  int64_t n, nboot, G;
  uint64_t seed;
  double lo[4], hi[4], h[4], denom, tmax;
  int64_t dims[4], stride[4], corner[16];
  const double *data;
  const int32_t *idx;
  uint32_t *cell, *pos, *cell_sorted, *cstart, *csum, *counts, *mult;
  double *rhs;  // remainders in cell order, N per sample
  unsigned long long *acc, *acc_lo;
  int *misc;  // error bits, largest count
};

namespace {

constexpr int kBT = 256;
constexpr int kScan = 2048;  // cells per block of the scan
constexpr int kDraws = 4;    // draws per thread
constexpr int kRes = 8;      // resamples per thread of the counts
constexpr int kMaxPer = 8, kConvPer = 4;

__host__ __device__ __forceinline__ int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

__device__ __forceinline__ double remainder_of(const BinJob &J, double x, int j) {
  return fmod(__dsub_rn(x, J.lo[j]), J.h[j]);
}

// Per sample: bounds check and lower cell (DirectSpace.jl:219-224), and its rank among the samples
// of the cell: lanes of a warp in one cell share an atomic (samples crowd into few cells where
// the tails are long: 4,000,000 samples on 128^3, 967 + 977 us for counts and ranks with an atomic each, about 200 so).
struct CellBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const int64_t s = block * (int64_t)kBT + threadIdx.x;
    const bool act = s < J.n;
    const unsigned lane = threadIdx.x & 31;
    int64_t c = 0;
    if (act) {
      bool bad_bound = false, bad_top = false;
      for (int j = 0; j < J.N; ++j) {
        const double x = J.data[s * J.N + j];
        if ((x >= J.hi[j]) | (x <= J.lo[j]) | !(x == x)) bad_bound = true;
        const double l = floor(__ddiv_rn(__dsub_rn(x, J.lo[j]), J.h[j]));
        if (!bad_bound && (l + 1.0 >= (double)J.dims[j] || l < 0.0)) bad_top = true;
        c += (bad_bound || bad_top ? 0 : (int64_t)l) * J.stride[j];
      }
      if (bad_bound) atomicOr(J.misc, 1);
      if (bad_top) atomicOr(J.misc, 2);
    }
    const unsigned long long key = act ? (unsigned long long)c : ~0ull - lane;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(same) - 1;
    uint32_t base = 0;
    if (act && (int)lane == leader) base = atomicAdd(J.counts + J.nboot * J.G + c, (uint32_t)__popc(same));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (act) {
      J.cell[s] = (uint32_t)c;
      J.pos[s] = base + __popc(same & ((1u << lane) - 1));
    }
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.n, kBT); }
};

__device__ __forceinline__ uint32_t block_add(uint32_t v, uint32_t *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  for (int w = 0; w < kBT / 32; ++w) t += sh[w];
  __syncthreads();
  return t;
}

// Sums of the cells' sample counts per block of kScan cells.
struct ChunkSumBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    __shared__ uint32_t sh[kBT / 32];
    const uint32_t *cnt = J.counts + J.nboot * J.G;
    const int64_t c0 = (int64_t)block * kScan;
    uint32_t v = 0;
    for (int k = threadIdx.x; k < kScan; k += kBT)
      if (c0 + k < J.G) v += cnt[c0 + k];
    v = block_add(v, sh);
    if (threadIdx.x == 0) J.csum[block] = v;
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.G, kScan); }
};

// cstart[c]: first position of cell c in cell order.  Each block adds up the sums before it.
struct StartBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    __shared__ uint32_t sh[kBT / 32];
    const uint32_t *cnt = J.counts + J.nboot * J.G;
    constexpr int PER = kScan / kBT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t before = 0;
    for (unsigned k = threadIdx.x; k < block; k += kBT) before += J.csum[k];
    before = block_add(before, sh);
    const int64_t c0 = (int64_t)block * kScan + threadIdx.x * PER;
    uint32_t v[PER], t = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      v[q] = c0 + q < J.G ? cnt[c0 + q] : 0u;
      t += v[q];
    }
    uint32_t scan = t;  // inclusive over the threads
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += u;
    }
    if (lane == 31) sh[warp] = scan;
    __syncthreads();
    uint32_t run = before + scan - t;
    for (int w = 0; w < warp; ++w) run += sh[w];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      if (c0 + q < J.G) J.cstart[c0 + q] = run;
      run += v[q];
    }
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.G, kScan); }
};

// Each sample's position in cell order, and there its cell and remainders.
struct PlaceBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const int64_t s = block * (int64_t)kBT + threadIdx.x;
    if (s >= J.n) return;
    const uint32_t c = J.cell[s], p = J.cstart[c] + J.pos[s];
    J.pos[s] = p;
    J.cell_sorted[p] = c;
    for (int j = 0; j < J.N; ++j) J.rhs[(int64_t)p * J.N + j] = remainder_of(J, J.data[s * J.N + j], j);
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.n, kBT); }
};

// mult[b n + position] = how often resample b draws the sample.  Bound by the random reads and
// atomics in the L2 (one resample's multiplicities stay there); four draws in flight a thread.
struct DrawBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const unsigned per = (unsigned)cdiv(J.n, kBT * kDraws), b = block / per;
    const int64_t j0 = (int64_t)(block - b * per) * (kBT * kDraws) + threadIdx.x;
    uint32_t *mult = J.mult + (int64_t)b * J.n;
    uint32_t p[kDraws];
#pragma unroll
    for (int u = 0; u < kDraws; ++u) {
      const int64_t j = j0 + u * kBT;
      if (j < J.n) {
        int64_t s;
        if (J.idx) {
          s = (int64_t)J.idx[(int64_t)b * J.n + j] - 1;
          if (s < 0 || s >= J.n) {
            atomicOr(J.misc, 4);
            s = 0;
          }
        } else {
          s = boot_draw(J.seed, J.n, b, j);
        }
        p[u] = J.pos[s];
      }
    }
#pragma unroll
    for (int u = 0; u < kDraws; ++u)
      if (j0 + u * kBT < J.n) atomicAdd(mult + p[u], 1u);
  }
  static int64_t blocks(const BinJob &J) { return J.nboot * cdiv(J.n, kBT * kDraws); }
};

// Runs of equal keys along the warp: same[k] whether the key 2^k lanes before is equal, last the
// run's last lane.
struct WarpRuns {
  bool same[5], last;
  __device__ __forceinline__ explicit WarpRuns(unsigned long long key) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, key, 1 << k);
      same[k] = lane >= (1 << k) && up == key;
    }
    last = __shfl_down_sync(0xffffffffu, key, 1) != key || lane == 31;
  }
  // the run's sum, in its last lane (keys that are equal lie side by side)
  template <class V>
  __device__ __forceinline__ V sum(V v) const {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const V u = __shfl_up_sync(0xffffffffu, v, 1 << k);
      if (same[k]) v += u;
    }
    return v;
  }
};

// counts[b G + cell]: draws of resample b in the cell, from the multiplicities in cell order: one
// atomic per run of a warp; the runs are found once for kRes resamples.
struct CountBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const unsigned per = (unsigned)cdiv(J.n, kBT), part = block / per;
    const int64_t i = (int64_t)(block - part * per) * kBT + threadIdx.x;
    const bool act = i < J.n;
    const int64_t b0 = (int64_t)part * kRes;
    const uint32_t c = act ? J.cell_sorted[i] : 0u;
    uint32_t m[kRes];
#pragma unroll
    for (int q = 0; q < kRes; ++q) m[q] = act && b0 + q < J.nboot ? J.mult[(b0 + q) * J.n + i] : 0u;
    const WarpRuns runs(act ? (unsigned long long)c : ~0ull - (threadIdx.x & 31));
#pragma unroll
    for (int q = 0; q < kRes; ++q) {
      const uint32_t v = runs.sum(m[q]);
      if (act && runs.last && v) atomicAdd(J.counts + (b0 + q) * J.G + c, v);
    }
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.nboot, kRes) * cdiv(J.n, kBT); }
};

// The largest count of any resample's cell (the samples' own included).
struct MaxBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const int64_t total = (J.nboot + 1) * J.G;
    uint32_t best = 0;
#pragma unroll
    for (int q = 0; q < kMaxPer; ++q) {
      const int64_t i = (int64_t)block * (kBT * kMaxPer) + q * kBT + threadIdx.x;
      if (i < total) best = max(best, J.counts[i]);
    }
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best > *(volatile unsigned *)(J.misc + 1))
      atomicMax(reinterpret_cast<unsigned *>(J.misc + 1), best);
  }
  static int64_t blocks(const BinJob &J) { return cdiv((J.nboot + 1) * J.G, kBT * kMaxPer); }
};

// The fixed-point exponents from the largest count: a cell sums at most 2^N cmax terms, each <=
// tmax (means) or tmax^2 (squares); e = 62 - the binary exponent of that bound, and L leaves
// the low parts (|lo| <= 2^(L-1) a term) of as many terms below 2^62.
struct Scales {
  int em, ev, L;
  __device__ __forceinline__ explicit Scales(const BinJob &J) {
    const double cmax = (double)(uint32_t)J.misc[1], nc = (double)(1 << J.N);
    const double bm = __dmul_rn(__dmul_rn(nc, cmax > 1.0 ? cmax : 1.0), J.tmax);
    const double bv = __dmul_rn(bm, J.tmax);
    int xm, xv;
    frexp(bm, &xm);
    frexp(bv, &xv);
    em = 62 - xm;
    ev = 62 - xv;
    const unsigned long long terms = (unsigned long long)(1 << J.N) * (unsigned long long)(cmax > 1.0 ? cmax : 1.0);
    L = 62 - (terms <= 1 ? 0 : 64 - __clzll((long long)(terms - 1)));
  }
};

// v 2^e = hi + f (hi the nearest integer, |f| <= 1/2, both exact), lo = f 2^L rounded.
__device__ __forceinline__ void split_term(double v, int e, int L, unsigned long long &hi, unsigned long long &lo) {
  const double x = ldexp(v, e);
  const double xr = rint(x);
  hi = (unsigned long long)xr;
  lo = (unsigned long long)__double2ll_rn(ldexp(x - xr, L));
}

// The term of corner c (axis j takes the lower cell iff bit N - 1 - j is set) of the sample at
// position i, in the reference's order of operations (DirectSpace.jl:227-237), as fixed-point parts:
// mean high, mean low, square high, square low.
__device__ __forceinline__ void corner_term(const BinJob &J, int N, int64_t i, int c, const Scales &S,
                                            unsigned long long (&t)[4]) {
  double pl = 1.0, ph = 1.0;
  bool fl = false, fh = false;
  for (int j = 0; j < N; ++j) {
    const double rh = J.rhs[i * N + j];
    if ((c >> (N - 1 - j)) & 1) {
      const double rl = __dsub_rn(J.h[j], rh);
      pl = fl ? __dmul_rn(pl, rl) : rl;
      fl = true;
    } else {
      ph = fh ? __dmul_rn(ph, rh) : rh;
      fh = true;
    }
  }
  const double term = __ddiv_rn(__dmul_rn(pl, ph), J.denom);
  split_term(term, S.em, S.L, t[0], t[1]);
  split_term(__dmul_rn(term, term), S.ev, S.L, t[2], t[3]);
}

// The samples themselves (multiplicity 1) into the last array: one atomic per run of equal cells
// of a warp and part.
struct SelfBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const int64_t i = (int64_t)block * kBT + threadIdx.x;
    const bool act = i < J.n;
    const Scales S(J);
    const uint32_t c0 = act ? J.cell_sorted[i] : 0u;
    const WarpRuns runs(act ? (unsigned long long)c0 : ~0ull - (threadIdx.x & 31));
    const int64_t o = 2 * ((J.nboot + 1) / 2) * J.G;
    for (int c = 0; c < (1 << J.N); ++c) {
      unsigned long long t[4] = {0, 0, 0, 0};
      if (act) corner_term(J, J.N, i, c, S, t);
      const unsigned long long hi = runs.sum(t[0]), lo = runs.sum(t[1]);
      if (act && runs.last) {
        const int64_t at = (o + c0 + J.corner[c]) * 2;
        if (hi) atomicAdd(J.acc + at, hi);
        if (lo) atomicAdd(J.acc_lo + at, lo);
      }
    }
  }
  static int64_t blocks(const BinJob &J) { return cdiv(J.n, kBT); }
};

// The resamples: a warp's lanes are 32 resamples, its samples (J.samples consecutive ones in cell
// order) pass one by one with their terms, the same for every lane, from shared memory; each lane
// adds multiplicity x term in registers and gives the sums of a cell to memory when the next
// sample's cell is another one.  The next cell along axis 1 shares half of the corners, whose sums
// stay.  (With lanes along the samples a warp needed a segmented shuffle scan of every part
// for every resample: 4,000,000 samples on 128^3, 32 resamples: 9.5 ms, and 3.8 ms to store the terms
// in cell order; 5.0 ms here.)  NC corners a pass; 4-D takes two.
constexpr int kWarps = 4;
template <int N>
struct ResampleBody {
  static constexpr int NC = N == 4 ? 8 : (1 << N), PASS = N == 4 ? 2 : 1;
  static constexpr int LOWX = NC / 2;  // corners with this bit of q take the lower cell of axis 1
  struct Smem {
    ulonglong4 term[kWarps][32][NC];
    uint32_t mult[kWarps][32][33];
    uint32_t cell[kWarps][32];
  };
  // resample groups of at most 32, as even as possible; warps of a block: gw groups x 4 / gw chunks
  __host__ __device__ static int groups(const BinJob &J) { return (int)cdiv(J.nboot, 32); }
  __host__ __device__ static int gwarps(int g) { return g >= 3 ? 4 : g; }
  __host__ __device__ static int64_t chunk_blocks(const BinJob &J) {
    return cdiv(cdiv(J.n, J.samples), kWarps / gwarps(groups(J)));
  }
  static int64_t blocks(const BinJob &J) {
    const int g = groups(J);
    return J.nboot ? chunk_blocks(J) * cdiv(g, gwarps(g)) * PASS : 0;
  }
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    extern __shared__ ulonglong4 smr[];
    Smem &sm = *reinterpret_cast<Smem *>(smr);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ng = groups(J), gw = gwarps(ng);
    const unsigned cb = (unsigned)chunk_blocks(J);
    const unsigned rest = block / cb, pass = rest % PASS, part = rest / PASS;
    const int team = warp / gw, group = (int)part * gw + warp % gw;
    const int64_t first = ((int64_t)(block - rest * cb) * (kWarps / gw) + team) * J.samples;
    const int per = (int)cdiv(J.nboot, ng);  // resamples of a group
    const int64_t g0 = (int64_t)group * per;
    const int64_t b = g0 + lane;
    const bool mine = group < ng && lane < per && b < J.nboot;
    const Scales S(J);
    auto corner_of = [&](int q) { return N == 4 ? 2 * q + (int)pass : q; };
    unsigned long long a[NC][4];
#pragma unroll
    for (int q = 0; q < NC; ++q)
#pragma unroll
      for (int k = 0; k < 4; ++k) a[q][k] = 0;
    const int64_t om = 2 * (b >> 1) * J.G, ov = om + J.G;
    const int half = (int)(b & 1);
    auto give = [&](int q, uint32_t cell) {
      if (mine) {
        const int64_t cc = (int64_t)cell + J.corner[corner_of(q)];
        const int64_t m = (om + cc) * 2 + half, v = (ov + cc) * 2 + half;
        if (a[q][0]) atomicAdd(J.acc + m, a[q][0]);
        if (a[q][1]) atomicAdd(J.acc_lo + m, a[q][1]);
        if (a[q][2]) atomicAdd(J.acc + v, a[q][2]);
        if (a[q][3]) atomicAdd(J.acc_lo + v, a[q][3]);
      }
    };
    uint32_t cur = 0xffffffffu;
    for (int s0 = 0; s0 < J.samples; s0 += 32) {  // the same trips in every warp
      const int64_t i0 = first + s0;
      const int count = (int)max((int64_t)0, min((int64_t)32, J.n - i0));
      for (int r = 0; r < 32; ++r) {
        const int64_t br = g0 + r;
        sm.mult[warp][r][lane] =
            group < ng && r < per && br < J.nboot && lane < count ? J.mult[br * J.n + i0 + lane] : 0u;
      }
      const int tt = (warp % gw) * 32 + lane;  // the team's threads share the terms
      for (int e = tt; e < 32 * NC; e += gw * 32) {
        const int i = e / NC, q = e - i * NC;
        unsigned long long t[4] = {0, 0, 0, 0};
        if (i < count) corner_term(J, N, i0 + i, corner_of(q), S, t);
        sm.term[team][i][q] = make_ulonglong4(t[0], t[1], t[2], t[3]);
      }
      if (tt < 32) sm.cell[team][tt] = tt < count ? J.cell_sorted[i0 + tt] : 0u;
      __syncthreads();
      for (int i = 0; i < count; ++i) {
        const uint32_t c = sm.cell[team][i];
        if (c != cur) {
          if (cur != 0xffffffffu) {
            const bool next = c == cur + 1;  // then the same row: a lower cell is never the row's last point
#pragma unroll
            for (int q = 0; q < LOWX; ++q) {
              give(q | LOWX, cur);
              if (!next) give(q, cur);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                a[q | LOWX][k] = next ? a[q][k] : 0;
                a[q][k] = 0;
              }
            }
          }
          cur = c;
        }
        const uint32_t m = sm.mult[warp][lane][i];
#pragma unroll
        for (int q = 0; q < NC; ++q) {
          const ulonglong4 t = sm.term[team][i][q];
          a[q][0] += (unsigned long long)m * t.x;
          a[q][1] += (unsigned long long)m * t.y;
          a[q][2] += (unsigned long long)m * t.z;
          a[q][3] += (unsigned long long)m * t.w;
        }
      }
      __syncthreads();
    }
    if (cur != 0xffffffffu) {
#pragma unroll
      for (int q = 0; q < NC; ++q) give(q, cur);
    }
  }
};

template <int N>
__global__ void __launch_bounds__(kWarps * 32)
    resample_kernel(const BinJob *jobs, const unsigned *block0, int count) {
  __shared__ BinJob job;
  unsigned first;
  find_job(jobs, block0, count, job, first);
  ResampleBody<N>::run(job, blockIdx.x - first);
}

// The sums as FP64, in place: hi 2^-e + lo 2^-(e+L) (arrays of squares use their exponent).
struct ConvertBody {
  static __device__ __forceinline__ void run(const BinJob &J, unsigned block) {
    const unsigned per = (unsigned)cdiv(2 * J.G, kBT * kConvPer), arr = block / per;
    const int64_t npairs = (J.nboot + 1) / 2;
    const Scales S(J);
    const double sc = ldexp(1.0, -(arr < 2 * npairs && (arr & 1) ? S.ev : S.em));
    const int64_t i0 = (int64_t)(block - arr * per) * (kBT * kConvPer) + threadIdx.x;
    unsigned long long *v = J.acc + (int64_t)arr * 2 * J.G;
    const unsigned long long *lo = J.acc_lo + (int64_t)arr * 2 * J.G;
#pragma unroll
    for (int q = 0; q < kConvPer; ++q) {
      const int64_t i = i0 + q * kBT;
      if (i < 2 * J.G) {
        const double xl = (double)(long long)lo[i];
        reinterpret_cast<double *>(v)[i] = fma(ldexp(xl, -S.L), sc, (double)v[i] * sc);
      }
    }
  }
  static int64_t blocks(const BinJob &J) { return (2 * ((J.nboot + 1) / 2) + 1) * cdiv(2 * J.G, kBT * kConvPer); }
};

size_t al(size_t x) { return (x + 255) & ~size_t(255); }

BinJob bin_job(const DiracJob &d) {
  const pkde_grid *g = d.g;
  BinJob J{};
  J.N = g->ndim;
  J.n = d.n;
  J.samples = d.n >= (1 << 18) ? 128 : 32;  // long runs of a cell, or enough warps
  J.nboot = d.nboot;
  J.G = grid_size(g);
  J.seed = d.seed;
  int64_t s = 1;
  double sp = g->h[0];
  for (int j = 0; j < J.N; ++j) {
    J.lo[j] = g->lo[j];
    J.hi[j] = g->hi[j];
    J.h[j] = g->h[j];
    J.dims[j] = g->dims[j];
    J.stride[j] = s;
    s *= g->dims[j];
    if (j) sp = sp * g->h[j];
  }
  for (int c = 0; c < (1 << J.N); ++c)
    for (int j = 0; j < J.N; ++j)
      if (!((c >> (J.N - 1 - j)) & 1)) J.corner[c] += J.stride[j];
  // term <= prod(h) / (n prod(h)^2)
  J.denom = (double)d.n * (sp * sp);
  J.tmax = (1.0 / ((double)d.n * sp)) * (1.0 + 1e-12);
  J.data = d.d_data;
  J.idx = d.d_idx;
  J.cell = d.cell;
  J.pos = d.pos;
  J.cell_sorted = d.cell_sorted;
  J.cstart = d.cstart;
  J.csum = d.csum;
  J.counts = d.counts;
  J.mult = d.mult;
  J.rhs = d.rhs;
  J.acc = reinterpret_cast<unsigned long long *>(d.paired_out);
  J.acc_lo = d.acc_lo;
  J.misc = d.misc;
  return J;
}

}  // namespace

// Memory that must be zero before binning_run: spectra, low parts, counts, multiplicities.
size_t dirac_zero_bytes(const pkde_grid *g, int64_t n, int64_t nboot) {
  const int64_t G = grid_size(g), arrays = 2 * ((nboot + 1) / 2) + 1;
  return 2 * al(sizeof(double2) * arrays * G) + al(sizeof(uint32_t) * (nboot + 1) * G) + al(sizeof(uint32_t) * nboot * n);
}
size_t dirac_job_scratch(const pkde_grid *g, int64_t n) {
  const int64_t G = grid_size(g);
  return 3 * al(sizeof(uint32_t) * n) + al(sizeof(double) * g->ndim * n) + al(sizeof(uint32_t) * G) +
         al(sizeof(uint32_t) * cdiv(G, kScan));
}
void dirac_job_bind(DiracJob &j, char *zero, char *scratch, int *misc) {
  const int64_t G = grid_size(j.g), arrays = 2 * ((j.nboot + 1) / 2) + 1;
  auto take = [](char *&p, size_t bytes) {
    char *q = p;
    p += al(bytes);
    return q;
  };
  j.paired_out = (double2 *)take(zero, sizeof(double2) * arrays * G);
  j.acc_lo = (unsigned long long *)take(zero, sizeof(double2) * arrays * G);
  j.counts = (uint32_t *)take(zero, sizeof(uint32_t) * (j.nboot + 1) * G);
  j.mult = (uint32_t *)zero;
  j.cell = (uint32_t *)take(scratch, sizeof(uint32_t) * j.n);
  j.pos = (uint32_t *)take(scratch, sizeof(uint32_t) * j.n);
  j.cell_sorted = (uint32_t *)take(scratch, sizeof(uint32_t) * j.n);
  j.rhs = (double *)take(scratch, sizeof(double) * j.g->ndim * j.n);
  j.cstart = (uint32_t *)take(scratch, sizeof(uint32_t) * G);
  j.csum = (uint32_t *)scratch;
  j.misc = misc;
}

// Kernels of a binning: the block prefixes of each, per set of jobs.
constexpr int kBinKernels = 13;

// Device descriptors of `count` jobs: the jobs ordered by dimension, then per kernel the first
// blocks of the jobs.
size_t binning_desc_bytes(int count) { return al(sizeof(BinJob) * count) + al(sizeof(unsigned) * kBinKernels * count); }

void binning_describe(const DiracJob *jobs, int count, void *host, BinningPlan &plan) {
  BinJob *hj = (BinJob *)host;
  unsigned *b0 = (unsigned *)((char *)host + al(sizeof(BinJob) * count));
  int k = 0;
  for (int N = 1; N <= 4; ++N) {
    plan.first[N - 1] = k;
    for (int e = 0; e < count; ++e) {
      if (jobs[e].g->ndim != N) continue;
      if (jobs[e].n < 1 || jobs[e].n >= (int64_t(1) << 31)) throw invalid("number of samples must be in [1, 2^31)");
      hj[k++] = bin_job(jobs[e]);
    }
  }
  plan.first[4] = k;
  plan.count = count;
  auto prefix = [&](int kernel, int from, int to, auto blocks) {
    int64_t at = 0;
    for (int e = from; e < to; ++e) {
      b0[kernel * count + e] = (unsigned)at;
      at += blocks(hj[e]);
    }
    if (at > 0x7fffffff) throw Error{PKDE_EUNSUPPORTED, "too many samples in one call"};
    plan.blocks[kernel] = (unsigned)at;
  };
  prefix(0, 0, count, CellBody::blocks);
  prefix(1, 0, count, ChunkSumBody::blocks);
  prefix(2, 0, count, StartBody::blocks);
  prefix(3, 0, count, PlaceBody::blocks);
  prefix(4, 0, count, DrawBody::blocks);
  prefix(5, 0, count, CountBody::blocks);
  prefix(6, 0, count, MaxBody::blocks);
  prefix(7, 0, count, SelfBody::blocks);
  prefix(8, plan.first[0], plan.first[1], ResampleBody<1>::blocks);
  prefix(9, plan.first[1], plan.first[2], ResampleBody<2>::blocks);
  prefix(10, plan.first[2], plan.first[3], ResampleBody<3>::blocks);
  prefix(11, plan.first[3], plan.first[4], ResampleBody<4>::blocks);
  prefix(12, 0, count, ConvertBody::blocks);
}

// The binning of the described jobs; their zero memory and misc words are zero, the descriptors at
// dev.  Error bits (misc[0]) are the caller's to read back and check (binning_flags_check).
void binning_run(pkde_ctx *ctx, const BinningPlan &plan, const void *dev, cudaStream_t st) {
  const BinJob *jobs = (const BinJob *)dev;
  const unsigned *b0 = (const unsigned *)((const char *)dev + al(sizeof(BinJob) * plan.count));
  auto launch = [&](int kernel, int from, int to, int threads, size_t smem, auto kern) {
    if (!plan.blocks[kernel]) return;
    if (smem) allow_dynamic_smem(ctx, kern, smem);
    {
      Trace tr(ctx, PKDE_PHASE_BINNING, st);
      kern<<<plan.blocks[kernel], threads, smem, st>>>(jobs + from, b0 + kernel * plan.count + from, to - from);
    }
    PKDE_CHECK_LAUNCH();
  };
  const int all = plan.count;
  launch(0, 0, all, kBT, 0, many_jobs_kernel<CellBody, BinJob, kBT>);
  launch(1, 0, all, kBT, 0, many_jobs_kernel<ChunkSumBody, BinJob, kBT>);
  launch(2, 0, all, kBT, 0, many_jobs_kernel<StartBody, BinJob, kBT>);
  launch(3, 0, all, kBT, 0, many_jobs_kernel<PlaceBody, BinJob, kBT>);
  launch(4, 0, all, kBT, 0, many_jobs_kernel<DrawBody, BinJob, kBT>);
  launch(5, 0, all, kBT, 0, many_jobs_kernel<CountBody, BinJob, kBT>);
  launch(6, 0, all, kBT, 0, many_jobs_kernel<MaxBody, BinJob, kBT>);
  launch(7, 0, all, kBT, 0, many_jobs_kernel<SelfBody, BinJob, kBT>);
  launch(8, plan.first[0], plan.first[1], kWarps * 32, sizeof(ResampleBody<1>::Smem), resample_kernel<1>);
  launch(9, plan.first[1], plan.first[2], kWarps * 32, sizeof(ResampleBody<2>::Smem), resample_kernel<2>);
  launch(10, plan.first[2], plan.first[3], kWarps * 32, sizeof(ResampleBody<3>::Smem), resample_kernel<3>);
  launch(11, plan.first[3], plan.first[4], kWarps * 32, sizeof(ResampleBody<4>::Smem), resample_kernel<4>);
  launch(12, 0, all, kBT, 0, many_jobs_kernel<ConvertBody, BinJob, kBT>);
}

void binning_flags_check(const int *hmisc) {
  if (hmisc[0] & 1) throw invalid("Data points lie beyond grid. Remove them or increase grid boundaries.");
  if (hmisc[0] & 2)
    throw invalid("Data points lie within one rounding of the upper grid bound. Remove them or increase grid boundaries.");
  if (hmisc[0] & 4) throw invalid("Bootstrap indices must lie in 1:n_samples.");
}

}  // namespace pkde
