// Job descriptors of the chunked bandwidth steps (pkde_chunk.cu, pkde_chunk_pow2.cu).
#pragma once

#include "pkde_lines.cuh"
#include "pkde_step.cuh"

namespace pkde {

// One grid axis.  Lines of n = R M points: R = 1, plain Stockham stages; R = 3 or 5 (M a power
// of two from 8), the R interleaved sub-lines x[R n2 + n1] through the stages of M, then
// one radix-R combine X[k2 + M q] = sum_n1 W_n^(n1 k2) Y_n1[k2] W_R^(n1 q) (the step
// engine's mixed-radix arithmetic).
struct ChunkAxis {
  int n, M, R, nst, inner, lines;
  int generic_first;   // the first stage has a generic radix: one more exchange
  int fused;           // the first stage's sums fuse the scaling of one operand (power-of-two register tiles)
  int fixed;           // a length with passes of its own (pkde_chunk_len.cuh)
  const double2 *twc;  // combine twiddles [n1 - 1][k2]
  const double2 *plain;  // (cos, sin)(2 pi m / n) of a line with a stage of another radix, else nullptr
  Stage1 st[kStages1];
};
// Lines of a tile: L (pitch PN where a tile holds lines), Lr = L R sub-lines (pitch P); size: units
// of one tile; H: half the lines, rounded up (stages of other radices, R = 1).
struct ChunkTile {
  int L, Lr, P, PN, size, H;
  FastDiv dL, dLr, dH;
};

struct ChunkRun {
  int N, G, A, a0, C, mean;  // A arrays from a0 per step, C steps from s0; mean: index of the means' array
  int64_t s0, tab_stride;
  const double *fz, *fw, *cw;
  double invG;
  int dims[4];
  int64_t aoff[4];
};

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
  int G, A, C, arr0, rt, pairs, b0, nboot, tiles;  // blocks: tiles x steps
  double inv_n;
  const double *vscale, *recip;
  const double2 *in;
  double2 *state;
  double *out;
};

// 1 / i for the running variance over bootstraps: a table of the IEEE quotients for i < kChunkRecip,
// read with an index that is the same for the block.
constexpr int kChunkRecip = 4096;
__device__ __forceinline__ double recip_of(const double *table, int i) {
  return i < kChunkRecip ? __ldg(table + i) : 1.0 / (double)i;
}

// VMR of the two bootstraps of a pair at one point (DirectSpace.jl:550-552), 1 / n as a product; mean: of
// the bootstraps before.  |V| / n is the fused product, as in the engine's tiles: where all resamples are alike, the
// variance over them is the rounding of the ratio itself.
__device__ __forceinline__ void chunk_vmr2(double2 z, double2 w, double inv_n, double mean, double &xa, double &xb) {
  const double ma = __dmul_rn(fabs(z.x), inv_n), mb = __dmul_rn(fabs(z.y), inv_n);
  div_nr2(__fma_rn(fabs(w.x), inv_n, -__dmul_rn(ma, ma)), ma, __fma_rn(fabs(w.y), inv_n, -__dmul_rn(mb, mb)), mb, mean,
          xa, xb);
}

__device__ __forceinline__ void chunk_welford(double x, double inv, double2 &st) {
  const double delta = __dsub_rn(x, st.x);
  st.x = __fma_rn(delta, inv, st.x);
  st.y = __fma_rn(delta, __dsub_rn(x, st.x), st.y);
}

// Passes along power-of-two axes (ax.fused, 16 to 1024 points) on register tiles
// (pkde_chunk_pow2.cu).
void chunk_pow2_axis(pkde_ctx *ctx, const AxisJob &J, bool spectra, cudaStream_t st);
void chunk_pow2_rows(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st);
void chunk_pow2_means(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st);

// Passes along axes of the lengths known at compile time (pkde_chunk_len.cuh).
bool chunk_len_known(int n, int R);
void chunk_len_axis(pkde_ctx *ctx, const AxisJob &J, bool spectra, cudaStream_t st);
void chunk_len_rows(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st);
void chunk_len_means(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st);

}  // namespace pkde
