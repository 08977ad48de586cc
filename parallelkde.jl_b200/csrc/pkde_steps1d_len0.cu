// 1-D steps of lengths 18 to 135.
#include "pkde_steps1d_len.cuh"

namespace pkde {

extern const OnePass kOnePasses0[kOneTable];
const OnePass kOnePasses0[kOneTable] = {
    one_pass<18>(), one_pass<20>(), one_pass<24>(), one_pass<25>(), one_pass<27>(), one_pass<30>(),
    one_pass<36>(), one_pass<40>(), one_pass<45>(), one_pass<48>(), one_pass<50>(), one_pass<54>(),
    one_pass<60>(), one_pass<72>(), one_pass<75>(), one_pass<80>(), one_pass<81>(), one_pass<90>(),
    one_pass<96>(), one_pass<100>(), one_pass<108>(), one_pass<120>(), one_pass<125>(), one_pass<135>(),
};

extern const OnePass kOnePasses1[kOneTable];
extern const OnePass kOnePasses2[kOneTable];
extern const OnePass kOnePasses3[kOneTable];
extern const OnePass kOnePasses4[kOneTable];

static const OnePass *find_one(int n) {
  const OnePass *tables[] = {kOnePasses0, kOnePasses1, kOnePasses2, kOnePasses3, kOnePasses4};
  for (const OnePass *t : tables)
    for (int i = 0; i < kOneTable; ++i)
      if (t[i].n == n) return t + i;
  return nullptr;
}

bool steps1d_len_known(int n) { return find_one(n) != nullptr; }
void steps1d_len_run(pkde_ctx *ctx, int n, const Job1 *jobs, int count, int S, cudaStream_t st) {
  find_one(n)->run(ctx, jobs, count, S, st);
}

}  // namespace pkde
