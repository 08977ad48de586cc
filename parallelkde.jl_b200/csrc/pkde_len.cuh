// Stockham stages of a 2^a 3^b 5^c length known at compile time: every stride, division and loop
// bound a constant.
#pragma once

#include "pkde_tile.cuh"

namespace pkde {

// The stages of make_plan for a 5-smooth length.
struct LenStages {
  int nst = 0, rad[10] = {};
};
__host__ __device__ constexpr LenStages len_stages(int m) {
  LenStages s;
  const int pref[5] = {8, 4, 2, 3, 5};
  for (int i = 0; i < 5; ++i)
    while (m % pref[i] == 0) {
      s.rad[s.nst++] = pref[i];
      m /= pref[i];
    }
  return s;
}

template <int n, int R>
struct Len {
  static constexpr int M = n / R;
  static constexpr LenStages S = len_stages(M);
  __host__ __device__ static constexpr int ns(int i) {
    int v = 1;
    for (int q = 0; q < i; ++q) v *= S.rad[q];
    return v;
  }
};

// One stage.  ld(l, j, v): the inputs of butterfly j of line l; st(l, pos, v): element pos + q Ns of line l
// is v[q].
template <int T, int M, int Q, int Ns, int Lr, class Ld, class St>
__device__ __forceinline__ void len_stage(const double2 *tw, Ld ld, St st) {
  constexpr int nb = M / Q, items = nb * Lr, IT = (items + T - 1) / T;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = (int)threadIdx.x + it * T;
    if ((it + 1) * T <= items || e < items) {
      const int j = e / Lr, l = e - j * Lr, jq = j / Ns;
      double2 v[Q];
      ld(l, j, v);
      if constexpr (Ns > 1) {
        const int k = j - jq * Ns;
        if (k > 0) {
          const double2 *w = tw + k * (Q - 1);
#pragma unroll
          for (int r = 1; r < Q; ++r) v[r] = cmul1(v[r], __ldg(w + r - 1));
        }
      }
      dft_r<Q>(v);
      st(l, j + jq * (Ns * (Q - 1)), v);
    }
  }
}

}  // namespace pkde
