// Host check of the stage tables of colore_gb300/csrc/fft.cuh: for every plan of
// fft_plans.h, a stage that takes its twiddles from its table gives the bits of
// one that takes them from the roots of unity, and the tables' length is tw_len.
#include <cstdio>
#include <cmath>
#include <cstring>
#include <vector>

#include "fft.cuh"
#include "fft_plans.h"

template <int L, int R, int r, int Ns, int S>
static int check_stage(const float2 *roots, const float4 *table)
{
  int bad = 0;
  for (int t = 0; t < L / R; t++) {
    float2 a[R], b[R];
    for (int i = 0; i < R; i++) a[i] = b[i] = make_float2(0.1f * i - t, 0.3f * t + i * i);
    cgfft::stage<L, R, r, Ns, S>(a, t, roots);
    cgfft::stage<L, R, r, Ns, S>(b, t, cgfft::StageTw{table});
    bad += memcmp(a, b, sizeof(a)) != 0;
  }
  return bad;
}

template <int L, int R, int r0, int r1, int r2>
static int check_plan()
{
  std::vector<float2> roots(L);
  for (int j = 0; j < L; j++)
    roots[j] = make_float2((float)cos(2 * M_PI * j / L), (float)sin(2 * M_PI * j / L));
  constexpr int n = cgfft::tw_len<r0, r1, r2>;
  const float mark = 77.0f;
  std::vector<float4> tab(n + 1, make_float4(mark, mark, mark, mark));
  cgfft::tw_build<L, r0, r1, r2>(roots.data(), tab.data());
  int bad = tab[n].x != mark || (n > 0 && tab[n - 1].w == mark);
  bad += check_stage<L, R, r1, r0, 1>(roots.data(), tab.data()) + check_stage<L, R, r1, r0, -1>(roots.data(), tab.data());
  if constexpr (r2 > 1)
    bad += check_stage<L, R, r2, r0 * r1, 1>(roots.data(), tab.data() + r0 * r1 / 2) +
           check_stage<L, R, r2, r0 * r1, -1>(roots.data(), tab.data() + r0 * r1 / 2);
  return bad;
}

template <int N>
static void check_size()
{
  using PL = Plan<N>;
  printf("%d %d\n", N,
         check_plan<N, PL::CR, PL::C0, PL::C1, PL::C2>() + check_plan<N, PL::FR, PL::F0, PL::F1, PL::F2>() +
             check_plan<N / 2, PL::RR, PL::R0, PL::R1, PL::R2>());
}

int main()
{
  check_size<64>();
  check_size<96>();
  check_size<128>();
  check_size<192>();
  check_size<256>();
  check_size<384>();
  check_size<512>();
  check_size<1024>();
  check_size<2048>();
  return 0;
}
