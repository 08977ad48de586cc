// Passes of lengths 18 to 90.
#include "pkde_chunk_len.cuh"

namespace pkde {

extern const LenPasses kLenPasses0[kLenTable];
const LenPasses kLenPasses0[kLenTable] = {
    len_passes<18>(), len_passes<20>(), len_passes<24>(), len_passes<25>(), len_passes<27>(), len_passes<30>(),
    len_passes<36>(), len_passes<40>(), len_passes<45>(), len_passes<48>(), len_passes<50>(), len_passes<54>(),
    len_passes<60>(), len_passes<72>(), len_passes<75>(), len_passes<80>(), len_passes<81>(), len_passes<90>(),
};

extern const LenPasses kLenPasses1[kLenTable];
extern const LenPasses kLenPasses2[kLenTable];
extern const LenPasses kLenPasses3[kLenTable];

static const LenPasses *find_len(int n, int R) {
  const LenPasses *tables[] = {kLenPasses0, kLenPasses1, kLenPasses2, kLenPasses3};
  for (const LenPasses *t : tables)
    for (int i = 0; i < kLenTable; ++i)
      if (t[i].n == n && t[i].R == R) return t + i;
  return nullptr;
}

bool chunk_len_known(int n, int R) { return find_len(n, R) != nullptr; }
void chunk_len_axis(pkde_ctx *ctx, const AxisJob &J, bool spectra, cudaStream_t st) {
  find_len(J.ax.n, J.ax.R)->axis(ctx, J, spectra, st);
  PKDE_CHECK_LAUNCH();
}
void chunk_len_rows(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
  find_len(J.ax.n, J.ax.R)->rows(ctx, J, st);
  PKDE_CHECK_LAUNCH();
}
void chunk_len_means(pkde_ctx *ctx, const RowsJob &J, cudaStream_t st) {
  find_len(J.ax.n, J.ax.R)->means(ctx, J, st);
  PKDE_CHECK_LAUNCH();
}

}  // namespace pkde
